// step_fp64.cu -- the plain FP64 Rayleigh-Benard time step as fused lane passes.
//
// One call of Integrate::update (src/navier/navier.rs:737-765) is decomposed
// into passes along y (lanes = rows, contiguous) and along x (lanes = columns).
// Linear operators acting on different axes commute, so each pass applies all
// the work that is local to its lanes; the reference's results are reproduced
// up to floating-point reassociation.
//
//  periodic (FourierR2c x Chebyshev):  Y1 -> X -> Y2            (3 launches)
//  box (Chebyshev x Chebyshev):        Y1 -> X1 -> Y2 -> X2 -> Y3 -> X3 -> Y4 -> X4 -> Y5
//
// Each launch takes a table of work items (case, first lane, lane count); a
// batch of cases is the same launch with a longer table.
#include "lane_ops.cuh"
#include "cvt.cuh"
#include "pdl.cuh"
#include "split_emit.cuh"
#include "per_device.h"
#include "prims.h"
#include "step_fp64.h"
#include "step_split.h"

#include <algorithm>

namespace rbc {
namespace dev {

static __device__ __forceinline__ void flag_nonfinite(unsigned int* status) { atomicOr(status, 1u); }

// load a lane set: lane l (0 <= l < 3*nr) = field (l / nr), row (r0 + l % nr)
template <class T>
__device__ void load_rows3(void* const f[3], int row_len, int r0, int nr, T* dst, int ld, int tid, int nth) {
  for (int idx = tid; idx < 3 * nr * row_len; idx += nth) {
    int l = idx / row_len, j = idx - l * row_len;
    int fi = l / nr, r = l - fi * nr;
    dst[l * ld + j] = static_cast<const T*>(f[fi])[(size_t)(r0 + r) * row_len + j];
  }
  __syncthreads();
}

// three lanes of n doubles, element k at base + k * stride of each array: the
// three loads of a thread are issued together
__device__ __forceinline__ void load_lanes3(const void* a, const void* b, const void* d, size_t base, int stride, int n,
                                            double* dst, int ld, int tid, int nth) {
  const double* pa = static_cast<const double*>(a) + base;
  const double* pb = static_cast<const double*>(b) + base;
  const double* pd = static_cast<const double*>(d) + base;
  for (int k = tid; k < n; k += nth) {
    const size_t o = (size_t)k * stride;
    const double va = __ldcg(pa + o), vb = __ldcg(pb + o), vd = __ldcg(pd + o);
    dst[k] = va;
    dst[ld + k] = vb;
    dst[2 * ld + k] = vd;
  }
}

// ============================================================================
// Y1: Y0_f = Ty^-1 Sy f,  Y1_f = Ty^-1 Dy Sy f   for f in (ux, uy, temp)
// ============================================================================
template <class T>
__global__ void __launch_bounds__(256) k_y1(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int r0 = w.y, nr = w.z;
  const int ny = c.ny, myc = c.myc, ld = c.ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  T* IN = reinterpret_cast<T*>(smem);
  T* O = IN + 3 * nr * ld;   // 3nr ortho lanes, followed by
  T* D = O + 3 * nr * ld;    // 3nr derivative lanes
  T* TMP = D + 3 * nr * ld;
  double2* WA = reinterpret_cast<double2*>(TMP + 3 * nr * ld + 2);
  WA = reinterpret_cast<double2*>((reinterpret_cast<size_t>(WA) + 15) & ~size_t(15));
  const int wld = c.cy.use_fft ? c.cy.L : 1;
  double2* WB = WA + (size_t)3 * nr * wld;
  void* f3[3] = {c.ux, c.uy, c.temp};
  load_rows3<T>(f3, myc, r0, nr, IN, ld, tid, nth);
  to_ortho<T>(c.ycd, IN, ld, O, ld, 3 * nr, tid, nth);
  cheb_diff<T>(c.odd, O, ld, D, ld, ny, 3 * nr, 1, TMP, ld, tid, nth);
  // inverse Chebyshev transform of O and D (6nr lanes, O and D contiguous)
  if (c.cy.use_fft) {
    if constexpr (sizeof(T) == 16) {
      dct1_fft_c(c.cy, false, (const double2*)O, ld, (double2*)O, ld, 3 * nr, WA, WB, wld, tid, nth);
      dct1_fft_c(c.cy, false, (const double2*)D, ld, (double2*)D, ld, 3 * nr, WA, WB, wld, tid, nth);
    } else {
      dct1_fft_r(c.cy, false, (const double*)O, ld, (double*)O, ld, 6 * nr, WA, WB, wld, tid, nth);
    }
  } else {
    dct1_dense<T>(c.cy, false, O, ld, TMP, ld, 3 * nr, tid, nth);
    for (int idx = tid; idx < 3 * nr * ny; idx += nth) {
      int l = idx / ny, k = idx - l * ny;
      O[l * ld + k] = TMP[l * ld + k];
    }
    __syncthreads();
    dct1_dense<T>(c.cy, false, D, ld, TMP, ld, 3 * nr, tid, nth);
    for (int idx = tid; idx < 3 * nr * ny; idx += nth) {
      int l = idx / ny, k = idx - l * ny;
      D[l * ld + k] = TMP[l * ld + k];
    }
    __syncthreads();
  }
  // store: yw[2f] = O lanes, yw[2f+1] = D lanes; row stride ny
  for (int idx = tid; idx < 6 * nr * ny; idx += nth) {
    int l = idx / ny, k = idx - l * ny;
    int which = l / (3 * nr), ll = l - which * 3 * nr;
    int fi = ll / nr, r = ll - fi * nr;
    const T* src = which ? D : O;
    static_cast<T*>(c.yw[2 * fi + which])[(size_t)(r0 + r) * ny + k] = src[ll * ld + k];
  }
}

size_t smem_y1(const CaseDev& c, int nr, bool cplx) {
  size_t es = cplx ? 16 : 8;
  size_t ld = c.ny + 1;
  size_t base = 4 * 3 * nr * ld * es + 2 * 8 + 16;
  size_t wld = c.cy.use_fft ? c.cy.L : 1;
  return base + 2 * (size_t)3 * nr * wld * 16 + 64;
}

// solid-mask damping of the convection products at physical point g
// (navier.rs:551-560, 579-584, 603-608): conv -= (-1/eta) mask w with
// w = ux, uy, and T + T_bc - value for the temperature (f = 2)
__device__ __forceinline__ double solid_damp(const CaseDev& c, int f, size_t g, double p, double u, double v, double t) {
  const double cm = c.solid_cm[g];
  const double w = f == 0 ? u : f == 1 ? v : (t + c.bc_v[g]) - c.solid_val[g];
  return p - cm * w;
}

// ============================================================================
// Periodic X pass: one column j of the Y arrays.
//  u = F^-1 Y0_ux, v = F^-1 Y0_uy;  for f: a = F^-1 (ik/s Y0_f), b = F^-1 Y1_f
//  P_f = u a + v b (+ u dbc/dx + v dbc/dy for temp);  Q_f = F P_f, rows < kx
//  With a solid mask a ninth lane carries T = F^-1 Y0_t for the damping term.
// ============================================================================
__global__ void __launch_bounds__(256) k_per_x(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y;
  const int mx = c.mx, nx = c.nx, ny = c.ny, M = c.fx.M;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  const bool solid = c.solid_cm != nullptr;
  const int NL = solid ? 9 : 8;
  extern __shared__ double2 smem[];
  const int ild = mx + 1;         // input lanes (complex)
  double2* IN = smem;             // NL lanes
  double2* WA = IN + NL * ild;    // NL lanes of M
  double2* WB = WA + NL * M;
  double* PH = reinterpret_cast<double*>(IN);  // physical lanes alias the inputs (NL x nx reals)
  // lane order: Y0u, Y0v, ikY0u, Y1u, ikY0v, Y1v, ikY0t, Y1t (, Y0t)
  for (int idx = tid; idx < NL * mx; idx += nth) {
    int l = idx / mx, k = idx - l * mx;
    int src = (l == 8) ? 4 : (l < 2) ? 2 * l : (l & 1 ? 2 * ((l - 2) >> 1) + 1 : 2 * ((l - 2) >> 1));
    double2 v = static_cast<const double2*>(c.yw[src])[(size_t)k * ny + j];
    if (l >= 2 && l < 8 && !(l & 1)) v = mul_ik(v, (double)k) * inv_asp;
    IN[l * ild + k] = v;
  }
  __syncthreads();
  c2r(c.fx, IN, ild, 1, PH, nx, NL, WA, WB, M, tid, nth);
  // products into lanes 2, 4, 6
  const double* bx = c.bc_dx;
  const double* by = c.bc_dy;
  for (int idx = tid; idx < 3 * nx; idx += nth) {
    int f = idx / nx, x = idx - f * nx;
    double u = PH[x], v = PH[nx + x];
    double a = PH[(2 + 2 * f) * nx + x], b = PH[(3 + 2 * f) * nx + x];
    double p = u * a + v * b;
    if (f == 2) {
      p = p + u * bx[(size_t)x * ny + j];
      p = p + v * by[(size_t)x * ny + j];
    }
    if (solid) p = solid_damp(c, f, (size_t)x * ny + j, p, u, v, PH[8 * nx + x]);
    PH[(2 + 2 * f) * nx + x] = p;
  }
  __syncthreads();
  double2* q = static_cast<double2*>(c.q[0]);
  r2c(c.fx, PH + 2 * nx, 2 * nx, q + j, c.kx * ny, ny, c.kx, 3, WA, WB, M, tid, nth);
}

size_t smem_per_x(const CaseDev& c) {
  const size_t nl = c.solid_cm ? 9 : 8;
  size_t ild = c.mx + 1;
  size_t in_bytes = std::max(nl * ild * 16, nl * c.nx * 8);
  return in_bytes + 2 * nl * (size_t)c.fx.M * 16 + 64;
}

// ============================================================================
// Periodic Y2 pass: one row i.  Convection DCT, right-hand sides, Helmholtz
// solves (Hholtz per row), divergence, Poisson row solve, projection and the
// pressure update (navier.rs:622-721).
// ============================================================================
// The ADI factors are the same for every lane.  Up to this length they are staged
// in shared memory: a pass then has one CTA per SM, and a factor loaded inside a
// recurrence costs its L2 latency (box 129^2: x2 25 -> 14 us, y3 28 -> 15 us).
// Longer lanes leave several CTAs per SM to cover it, and the staging would cost
// one of them.  Box step, us, staged | not: 129^2 138.4 | 139.3, 200^2 184.7 |
// 186.6, 264^2 228.1 | 229.7, 300^2 242.4 | 245.4, 320^2 258.2 | 259.2, 360^2
// 296.9 | 298.8, 450^2 369.1 | 371.2, 513^2 497.0 | 474.7.  The line lies where
// the gain has become half a percent.
__host__ __device__ inline bool stage_factors(int m) { return m <= 320; }

// stage the factors of row `row` of a per-row banded solver into shared memory
__device__ FdmaDev stage_fdma_row(const FdmaDev& f, int row, double* dst, int tid, int nth) {
  const int m = f.m;
  const size_t off = (f.rows > 1) ? (size_t)row * f.stride : 0;
  const double* __restrict__ low = f.low + off;
  const double* __restrict__ dinv = f.dinv + off;
  const double* __restrict__ up1 = f.up1 + off;
  const double* __restrict__ up2 = f.up2 + off;
  for (int k = tid; k < m; k += nth) {
    const double a = __ldg(low + k), b = __ldg(dinv + k), u = __ldg(up1 + k), v = __ldg(up2 + k);
    dst[k] = a;
    dst[m + k] = b;
    dst[2 * m + k] = u;
    dst[3 * m + k] = v;
  }
  FdmaDev r = f;
  r.rows = 1;
  r.stride = 0;
  r.low = dst;
  r.dinv = dst + m;
  r.up1 = dst + 2 * m;
  r.up2 = dst + 3 * m;
  r.scan = f.scan + (f.rows > 1 ? (size_t)row * kFdmaScan : 0);
  return r;
}

// CONV: where the convection term comes from
//   CONV_Q      q, transformed along y here
//   CONV_MIXED  m_cv, transformed (the mixed form's GEMM), without the linear
//               boundary part (CaseDev::m_bclin)
//   CONV_FULL   m_cv, transformed and complete (the split GEMMs)
// Registers (BOUND: CTAs per SM they have to allow): left to itself the compiler
// takes 118, so that two CTAs of 256 threads fill an SM.  One case, with about two
// rows per SM, is fastest so.  The rows of a batch want four CTAs (64 registers,
// some spills), or three (80, none) where their shared memory allows only two;
// and the other group's passes, on their own branch of the graph, need registers
// beside them: at 118 a batch of both kinds took longer than its groups one after
// the other.  us per step, 118 | held: one case of 512 x 257 171.9 | 172.6 (80), 600 x
// 300 213 | 217 (80); four of 512 x 257, mixed 385 | 393 (80); 16 x (200 x 150)
// 506 | 420 (64), 32 x (128 x 128) 602 | 509 (64); mixed 64 x (128 x 65) 568 | 391 (64);
// mixed ensembles of 48, 64 and 128 cases 1248 | 985, 1505 | 1210, 2189 | 1929 (80).  The
// CTAs of 128 threads: 32 x (128 x 65) 203 | 169 (72).  CONV_Q is always held to 64 (8
// cases of 128 x 65: 76 us at 80 registers, 54).
enum { CONV_Q = 0, CONV_MIXED = 1, CONV_FULL = 2 };
template <int CONV, int NT = 256, int BOUND = 1>
__global__ void __launch_bounds__(NT, BOUND) k_per_y2(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  constexpr bool PRE = CONV != CONV_Q;
  const int i = w.y;
  const int ny = c.ny, myc = c.myc, kx = c.kx, ky = c.ky;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double dt = c.dt, nu = c.nu, inv_asp = 1.0 / c.aspect, ki = (double)i;
  extern __shared__ double2 smem[];
  double2* CV = smem;        // 3 lanes conv
  double2* REG = CV + 3 * ld;
  // during the convection transform REG holds the FFT work lanes; afterwards:
  double2* F = REG;          // 3 lanes composite state (old, then new)
  double2* O = F + 3 * ld;   // 3 lanes
  // rhs lanes (lane 0 later: divergence); with the convection term given (PRE)
  // they overwrite the convection lanes, which are dead once the rhs is formed
  double2* R = PRE ? CV : O + 3 * ld;
  double2* P = PRE ? O + 3 * ld : R + 3 * ld;  // p0 row
  double2* G = P + ld;       // d/dy
  double2* X1 = G + ld;      // 3 lanes
  const int wld = c.cy.use_fft ? c.cy.L : 1;
  double2* WA = REG;
  double2* WB = WA + 3 * wld;
  const size_t reg_elems = PRE ? (size_t)11 * ld : max((size_t)14 * ld, (size_t)6 * wld);
  double* FAC = reinterpret_cast<double*>(REG + reg_elems);
  // per-row factors of the three banded solves
  const FdmaDev fu = stage_fdma_row(c.hu_y, i, FAC, tid, nth);
  const FdmaDev ft = stage_fdma_row(c.ht_y, i, FAC + 4 * myc, tid, nth);
  const FdmaDev fp = stage_fdma_row(c.pois_y, i, FAC + 8 * myc, tid, nth);

  // 1. convection: forward Chebyshev transform of Q_f[i], dealiased
  if (PRE) {
    const double2* cv = static_cast<const double2*>(c.m_cv);
    for (int idx = tid; idx < 3 * ny; idx += nth) {
      int f = idx / ny, k = idx - f * ny;
      CV[f * ld + k] = (i < kx && k < ky) ? cv[((size_t)f * kx + i) * ky + k] : c2(0.0, 0.0);
    }
  } else if (i < kx) {
    const double2* q = static_cast<const double2*>(c.q[0]);
    for (int idx = tid; idx < 3 * ny; idx += nth) {
      int f = idx / ny, k = idx - f * ny;
      CV[f * ld + k] = q[(size_t)f * kx * ny + (size_t)i * ny + k];
    }
    __syncthreads();
    if (c.cy.use_fft) dct1_fft_c(c.cy, true, CV, ld, CV, ld, 3, WA, WB, wld, tid, nth);
    else {
      dct1_dense<double2>(c.cy, true, CV, ld, REG, ld, 3, tid, nth);
      for (int idx = tid; idx < 3 * ny; idx += nth) {
        int f = idx / ny, k = idx - f * ny;
        CV[f * ld + k] = REG[f * ld + k];
      }
      __syncthreads();
    }
    for (int idx = tid; idx < 3 * ny; idx += nth) {
      int f = idx / ny, k = idx - f * ny;
      if (k >= ky) CV[f * ld + k] = c2(0.0, 0.0);
    }
  } else {
    for (int idx = tid; idx < 3 * ny; idx += nth) CV[(idx / ny) * ld + idx % ny] = c2(0.0, 0.0);
  }
  __syncthreads();
  // 2. right-hand sides
  void* f3[3] = {c.ux, c.uy, c.temp};
  for (int idx = tid; idx < 3 * myc; idx += nth) {
    int f = idx / myc, k = idx - f * myc;
    F[f * ld + k] = static_cast<const double2*>(f3[f])[(size_t)i * myc + k];
  }
  const double2* p0 = static_cast<const double2*>(c.p0);
  for (int k = tid; k < ny; k += nth) P[k] = p0[(size_t)i * ny + k];
  __syncthreads();
  to_ortho<double2>(c.ycd, F, ld, O, ld, 3, tid, nth);
  cheb_diff<double2>(c.odd, P, ld, G, ld, ny, 1, 1, nullptr, ld, tid, nth);
  const double2* bco = static_cast<const double2*>(c.bc_ortho);
  const double2* bcd = static_cast<const double2*>(c.bc_diff);
  for (int k = tid; k < ny; k += nth) {
    double2 gx = mul_ik(P[k], ki) * inv_asp;
    double2 cu = CV[k], cvv = CV[ld + k], ct = CV[2 * ld + k];
    if (CONV == CONV_MIXED && c.m_bclin && i < kx && k < ky) ct = add_bclin(ct, O[ld + k], c.m_bcg, i);
    R[k] = fnms(fnms(O[k], gx, dt), cu, dt);
    double2 that = O[2 * ld + k] + bco[(size_t)i * ny + k];
    R[ld + k] = fnms(fmas(fnms(O[ld + k], G[k], dt), that, dt), cvv, dt);
    R[2 * ld + k] = fnms(O[2 * ld + k] + bcd[(size_t)i * ny + k], ct, dt);
  }
  __syncthreads();
  // 3. Helmholtz: pinv_y then the row's banded solve
  matvec_pinv<double2>(c.pinv_y, R, ld, F, ld, 3, tid, nth);
  // ux*, uy* (factors fu) and temp (factors ft): 6 chains in one phase
  fdma_solve2<double2>(fu, ft, 2, F, ld, 3, 0, 0, tid, nth);
  // 4. divergence = ik/s Sy ux* + Dy Sy uy*
  to_ortho<double2>(c.ycd, F, ld, O, ld, 2, tid, nth);
  cheb_diff<double2>(c.odd, O + ld, ld, G, ld, ny, 1, 1, nullptr, ld, tid, nth);
  for (int k = tid; k < ny; k += nth) R[k] = mul_ik(O[k], ki) * inv_asp + G[k];  // R lane 0 = div
  __syncthreads();
  // 5. Poisson row solve -> pseudo pressure row
  matvec_pinv<double2>(c.pinv_y, R, ld, X1, ld, 1, tid, nth);
  fdma_solve<double2>(fp, X1, ld, 1, 0, 0, tid, nth);
  if (i == 0 && tid == 0) X1[0] = c2(0.0, 0.0);
  __syncthreads();
  double2* p1 = static_cast<double2*>(c.p1);
  for (int k = tid; k < myc; k += nth) p1[(size_t)i * myc + k] = X1[k];
  // 6. projection: O1 = Sy^N p1; dpdx = ik/s O1; dpdy = Dy O1
  to_ortho<double2>(c.ycn, X1, ld, O, ld, 1, tid, nth);  // O lane 0 = O1
  cheb_diff<double2>(c.odd, O, ld, G, ld, ny, 1, 1, nullptr, ld, tid, nth);  // G = dpdy
  for (int k = tid; k < ny; k += nth) {
    O[ld + k] = mul_ik(O[k], ki) * inv_asp;  // O lane 1 = dpdx
    O[2 * ld + k] = G[k];                     // O lane 2 = dpdy
  }
  __syncthreads();
  from_ortho<double2>(c.ycd, O + ld, ld, X1 + ld, ld, 2, tid, nth);  // X1 lanes 1, 2
  // 7. pressure update and stores
  double2* pw = static_cast<double2*>(c.p0);
  for (int k = tid; k < ny; k += nth) {
    double2 v = fnms(P[k], R[k], nu);
    pw[(size_t)i * ny + k] = fmas(v, O[k], c.inv_dt);
  }
  double2* ux = static_cast<double2*>(c.ux);
  double2* uy = static_cast<double2*>(c.uy);
  double2* tt = static_cast<double2*>(c.temp);
  bool bad = false;
  for (int k = tid; k < myc; k += nth) {
    double2 a = F[k] - X1[ld + k];
    double2 b = F[ld + k] - X1[2 * ld + k];
    double2 t = F[2 * ld + k];
    ux[(size_t)i * myc + k] = a;
    uy[(size_t)i * myc + k] = b;
    tt[(size_t)i * myc + k] = t;
    bad |= !(finite_v(a) && finite_v(b) && finite_v(t));
  }
  if (bad) flag_nonfinite(c.status);
}

// ============================================================================
// Periodic Y2 split in two launches for more CTAs per SM:
//  Y2a (row i, field f): convection transform, right-hand side, pinv_y and the
//       row's banded Helmholtz solve; writes ux*, uy* (into the state arrays,
//       overwritten by Y2b) and the new temperature.
//  Y2b (row i): divergence, Poisson row solve, projection, pressure update.
// ============================================================================
__global__ void __launch_bounds__(256) k_per_y2a(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int i = w.y, f = w.w;
  const int ny = c.ny, myc = c.myc, kx = c.kx, ky = c.ky;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double dt = c.dt, inv_asp = 1.0 / c.aspect, ki = (double)i;
  extern __shared__ double2 smem[];
  double2* CV = smem;   // conv lane
  double2* REG = CV + ld;
  double2* F = REG;      // composite row of field f
  double2* T2 = F + ld;  // composite temperature row (buoyancy of uy)
  double2* O = T2 + ld;  // ortho of F
  double2* OT = O + ld;  // ortho of T2
  double2* R = OT + ld;  // rhs
  double2* P = R + ld;   // p0 row
  double2* G = P + ld;   // d/dy p0
  const int wld = c.cy.use_fft ? c.cy.L : 1;
  double2* WA = REG;
  double2* WB = WA + wld;
  const size_t reg_elems = max((size_t)7 * ld, (size_t)2 * wld);
  double* FAC = reinterpret_cast<double*>(REG + reg_elems);
  const FdmaDev fr = stage_fdma_row(f == 2 ? c.ht_y : c.hu_y, i, FAC, tid, nth);
  void* f3[3] = {c.ux, c.uy, c.temp};
  // convection
  if (i < kx) {
    const double2* q = static_cast<const double2*>(c.q[0]) + (size_t)f * kx * ny + (size_t)i * ny;
    for (int k = tid; k < ny; k += nth) CV[k] = q[k];
    __syncthreads();
    if (c.cy.use_fft) dct1_fft_c(c.cy, true, CV, ld, CV, ld, 1, WA, WB, wld, tid, nth);
    else {
      dct1_dense<double2>(c.cy, true, CV, ld, REG, ld, 1, tid, nth);
      for (int k = tid; k < ny; k += nth) CV[k] = REG[k];
      __syncthreads();
    }
    for (int k = tid; k < ny; k += nth)
      if (k >= ky) CV[k] = c2(0.0, 0.0);
  } else {
    for (int k = tid; k < ny; k += nth) CV[k] = c2(0.0, 0.0);
  }
  __syncthreads();
  // right-hand side
  const double2* st = static_cast<const double2*>(f3[f]) + (size_t)i * myc;
  for (int k = tid; k < myc; k += nth) F[k] = st[k];
  const double2* p0 = static_cast<const double2*>(c.p0) + (size_t)i * ny;
  if (f < 2)
    for (int k = tid; k < ny; k += nth) P[k] = p0[k];
  if (f == 1) {
    const double2* tt = static_cast<const double2*>(c.temp) + (size_t)i * myc;
    for (int k = tid; k < myc; k += nth) T2[k] = tt[k];
  }
  __syncthreads();
  to_ortho<double2>(c.ycd, F, ld, O, ld, f == 1 ? 2 : 1, tid, nth);  // O (and OT for uy)
  if (f == 1) cheb_diff<double2>(c.odd, P, ld, G, ld, ny, 1, 1, nullptr, ld, tid, nth);
  const double2* bco = static_cast<const double2*>(c.bc_ortho) + (size_t)i * ny;
  const double2* bcd = static_cast<const double2*>(c.bc_diff) + (size_t)i * ny;
  for (int k = tid; k < ny; k += nth) {
    double2 r;
    if (f == 0) {
      double2 gx = mul_ik(P[k], ki) * inv_asp;
      r = fnms(fnms(O[k], gx, dt), CV[k], dt);
    } else if (f == 1) {
      double2 that = OT[k] + bco[k];
      r = fnms(fmas(fnms(O[k], G[k], dt), that, dt), CV[k], dt);
    } else {
      r = fnms(O[k] + bcd[k], CV[k], dt);
    }
    R[k] = r;
  }
  __syncthreads();
  matvec_pinv<double2>(c.pinv_y, R, ld, F, ld, 1, tid, nth);
  fdma_solve<double2>(fr, F, ld, 1, 0, 0, tid, nth);
  // ux*, uy* go to the state arrays (Y2b overwrites them with the projected
  // fields); the new temperature goes to scratch yw[0] because the uy work of
  // the same row still reads the old temperature for the buoyancy.
  double2* out = (f == 2 ? static_cast<double2*>(c.yw[0]) : static_cast<double2*>(f3[f])) + (size_t)i * myc;
  bool bad = false;
  for (int k = tid; k < myc; k += nth) {
    double2 v = F[k];
    out[k] = v;
    bad |= !finite_v(v);
  }
  if (bad) flag_nonfinite(c.status);
}

size_t smem_per_y2a(const CaseDev& c) {
  size_t ld = c.ny + 1;
  size_t wld = c.cy.use_fft ? c.cy.L : 1;
  size_t reg = std::max((size_t)7 * ld, (size_t)2 * wld);
  return (ld + reg) * 16 + (size_t)4 * c.myc * 8 + 64;
}

__global__ void __launch_bounds__(256) k_per_y2b(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int i = w.y;
  const int ny = c.ny, myc = c.myc;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double nu = c.nu, inv_asp = 1.0 / c.aspect, ki = (double)i;
  extern __shared__ double2 smem[];
  double2* F = smem;       // 2 lanes: ux*, uy*
  double2* O = F + 2 * ld; // 3 lanes
  double2* R = O + 3 * ld; // divergence
  double2* G = R + ld;
  double2* X1 = G + ld;    // 3 lanes
  double* FAC = reinterpret_cast<double*>(X1 + 3 * ld);
  const FdmaDev fp = stage_fdma_row(c.pois_y, i, FAC, tid, nth);
  double2* ux = static_cast<double2*>(c.ux) + (size_t)i * myc;
  double2* uy = static_cast<double2*>(c.uy) + (size_t)i * myc;
  for (int k = tid; k < myc; k += nth) {
    F[k] = ux[k];
    F[ld + k] = uy[k];
  }
  __syncthreads();
  to_ortho<double2>(c.ycd, F, ld, O, ld, 2, tid, nth);
  cheb_diff<double2>(c.odd, O + ld, ld, G, ld, ny, 1, 1, nullptr, ld, tid, nth);
  for (int k = tid; k < ny; k += nth) R[k] = mul_ik(O[k], ki) * inv_asp + G[k];
  __syncthreads();
  matvec_pinv<double2>(c.pinv_y, R, ld, X1, ld, 1, tid, nth);
  fdma_solve<double2>(fp, X1, ld, 1, 0, 0, tid, nth);
  if (i == 0 && tid == 0) X1[0] = c2(0.0, 0.0);
  __syncthreads();
  double2* p1 = static_cast<double2*>(c.p1) + (size_t)i * myc;
  for (int k = tid; k < myc; k += nth) p1[k] = X1[k];
  to_ortho<double2>(c.ycn, X1, ld, O, ld, 1, tid, nth);
  cheb_diff<double2>(c.odd, O, ld, G, ld, ny, 1, 1, nullptr, ld, tid, nth);
  for (int k = tid; k < ny; k += nth) {
    O[ld + k] = mul_ik(O[k], ki) * inv_asp;
    O[2 * ld + k] = G[k];
  }
  __syncthreads();
  from_ortho<double2>(c.ycd, O + ld, ld, X1 + ld, ld, 2, tid, nth);
  double2* pw = static_cast<double2*>(c.p0) + (size_t)i * ny;
  for (int k = tid; k < ny; k += nth) {
    double2 v = fnms(pw[k], R[k], nu);
    pw[k] = fmas(v, O[k], c.inv_dt);
  }
  const double2* tn = static_cast<const double2*>(c.yw[0]) + (size_t)i * myc;
  double2* tt = static_cast<double2*>(c.temp) + (size_t)i * myc;
  bool bad = false;
  for (int k = tid; k < myc; k += nth) {
    double2 a = F[k] - X1[ld + k];
    double2 b = F[ld + k] - X1[2 * ld + k];
    ux[k] = a;
    uy[k] = b;
    tt[k] = tn[k];
    bad |= !(finite_v(a) && finite_v(b));
  }
  if (bad) flag_nonfinite(c.status);
}

size_t smem_per_y2b(const CaseDev& c) {
  size_t ld = c.ny + 1;
  return (size_t)10 * ld * 16 + (size_t)4 * c.myc * 8 + 64;
}

size_t smem_per_y2(const CaseDev& c) {
  size_t ld = c.ny + 1;
  size_t wld = c.cy.use_fft ? c.cy.L : 1;
  size_t reg = std::max((size_t)14 * ld, (size_t)6 * wld);
  return (3 * ld + reg) * 16 + (size_t)12 * c.myc * 8 + 64;
}
// with the convection term given: the rhs lanes reuse the convection lanes
size_t smem_per_y2_pre(const CaseDev& c) {
  size_t ld = c.ny + 1;
  return (3 * ld + 11 * ld) * 16 + (size_t)12 * c.myc * 8 + 64;
}

// ============================================================================
// Box passes (Chebyshev in x).  Real data.
// ============================================================================
// X1: columns j < ny.  x-backward of the y-transformed state, products,
// x-forward of the products (rows < kx), and d/dx p0.
__global__ void __launch_bounds__(256) k_box_x1(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y;
  const int nx = c.nx, ny = c.ny, mxc = c.mxc, kx = c.kx;
  const int ld = nx + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  const bool solid = c.solid_cm != nullptr;
  const int NL = solid ? 9 : 8;
  extern __shared__ double2 smem[];
  double* IN = reinterpret_cast<double*>(smem);  // NL lanes composite-x (mxc)
  double* OR = IN + NL * ld;                     // NL ortho lanes (nx)
  double* PH = OR + NL * ld;                     // NL physical lanes
  double* TMP = PH + NL * ld;                    // NL lanes
  double2* WA = reinterpret_cast<double2*>(TMP + NL * ld + 2);
  WA = reinterpret_cast<double2*>((reinterpret_cast<size_t>(WA) + 15) & ~size_t(15));
  const int wld = c.cx.use_fft ? c.cx.L : 1;
  double2* WB = WA + ((NL + 1) >> 1) * wld;
  // lanes: 0 Y0u, 1 Y0v, 2 Y0u(dx), 3 Y1u, 4 Y0v(dx), 5 Y1v, 6 Y0t(dx), 7 Y1t (, 8 Y0t)
  for (int idx = tid; idx < NL * mxc; idx += nth) {
    int l = idx / mxc, k = idx - l * mxc;
    int src = (l == 8) ? 4 : (l < 2) ? 2 * l : (l & 1 ? 2 * ((l - 2) >> 1) + 1 : 2 * ((l - 2) >> 1));
    IN[l * ld + k] = static_cast<const double*>(c.yw[src])[(size_t)k * ny + j];
  }
  __syncthreads();
  // x stencils: lanes 0-5 use the velocity basis, 6-8 the temperature basis
  to_ortho<double>(c.xu, IN, ld, OR, ld, 6, tid, nth);
  to_ortho<double>(c.xt, IN + 6 * ld, ld, OR + 6 * ld, ld, NL - 6, tid, nth);
  // d/dx for lanes 2, 4, 6 (in place through TMP)
  cheb_diff<double>(c.odd, OR + 2 * ld, 2 * ld, TMP, ld, nx, 3, 1, nullptr, 0, tid, nth);
  for (int f = 0; f < 3; f++)
    for (int k = tid; k < nx; k += nth) OR[(2 + 2 * f) * ld + k] = TMP[f * ld + k] * inv_asp;
  __syncthreads();
  if (c.cx.use_fft) dct1_fft_r(c.cx, false, OR, ld, PH, ld, NL, WA, WB, wld, tid, nth);
  else dct1_dense<double>(c.cx, false, OR, ld, PH, ld, NL, tid, nth);
  // products (lanes 2, 4, 6)
  for (int idx = tid; idx < 3 * nx; idx += nth) {
    int f = idx / nx, x = idx - f * nx;
    double u = PH[x], v = PH[ld + x];
    double p = u * PH[(2 + 2 * f) * ld + x] + v * PH[(3 + 2 * f) * ld + x];
    if (f == 2) {
      p = p + u * c.bc_dx[(size_t)x * ny + j];
      p = p + v * c.bc_dy[(size_t)x * ny + j];
    }
    if (solid) p = solid_damp(c, f, (size_t)x * ny + j, p, u, v, PH[8 * ld + x]);
    TMP[f * ld + x] = p;
  }
  __syncthreads();
  // forward x transform of the 3 products -> OR lanes 0..2
  if (c.cx.use_fft) dct1_fft_r(c.cx, true, TMP, ld, OR, ld, 3, WA, WB, wld, tid, nth);
  else dct1_dense<double>(c.cx, true, TMP, ld, OR, ld, 3, tid, nth);
  double* q = static_cast<double*>(c.q[0]);
  for (int idx = tid; idx < 3 * kx; idx += nth) {
    int f = idx / kx, k = idx - f * kx;
    q[(size_t)f * kx * ny + (size_t)k * ny + j] = OR[f * ld + k];
  }
  // d/dx p0 column / aspect -> s[0] (nx x ny)
  const double* p0 = static_cast<const double*>(c.p0);
  for (int k = tid; k < nx; k += nth) IN[k] = p0[(size_t)k * ny + j];
  __syncthreads();
  cheb_diff<double>(c.odd, IN, ld, TMP, ld, nx, 1, 1, TMP + ld, ld, tid, nth);
  double* gp = static_cast<double*>(c.s[0]);
  for (int k = tid; k < nx; k += nth) gp[(size_t)k * ny + j] = TMP[k] * inv_asp;
}

// d/dx p0 / aspect for column j -> s[0] (nx x ny): the pressure-gradient part
// of X1, run on its own in the mixed-precision step (FP64)
__global__ void __launch_bounds__(256) k_box_gpx(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y;
  const int nx = c.nx, ny = c.ny;
  const int ld = nx + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  extern __shared__ double2 smem[];
  double* IN = reinterpret_cast<double*>(smem);
  double* TMP = IN + ld;
  const double* p0 = static_cast<const double*>(c.p0);
  for (int k = tid; k < nx; k += nth) IN[k] = p0[(size_t)k * ny + j];
  __syncthreads();
  cheb_diff<double>(c.odd, IN, ld, TMP, ld, nx, 1, 1, TMP + ld, ld, tid, nth);
  double* gp = static_cast<double*>(c.s[0]);
  for (int k = tid; k < nx; k += nth) gp[(size_t)k * ny + j] = TMP[k] * inv_asp;
}

size_t smem_box_gpx(const CaseDev& c) { return 3 * (size_t)(c.nx + 1) * 8 + 64; }

size_t smem_box_x1(const CaseDev& c) {
  const size_t nl = c.solid_cm ? 9 : 8;
  size_t ld = c.nx + 1;
  size_t wld = c.cx.use_fft ? c.cx.L : 1;
  return 4 * nl * ld * 8 + 2 * ((nl + 1) / 2) * wld * 16 + 64;
}

// Y2: rows i < nx (ortho x).  conv (y forward, dealiased), rhs, pinv_y -> s[1..3]
template <int CONV>
__global__ void __launch_bounds__(256) k_box_y2(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  constexpr bool PRE = CONV != CONV_Q;
  const int i = w.y;
  const int nx = c.nx, ny = c.ny, myc = c.myc, kx = c.kx, ky = c.ky, mxc = c.mxc;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double dt = c.dt;
  extern __shared__ double2 smem[];
  double* CV = reinterpret_cast<double*>(smem);  // 3 lanes
  double* SX = CV + 3 * ld;   // 3 lanes: Sx f (composite y)
  double* O = SX + 3 * ld;    // 3 lanes
  double* R = O + 3 * ld;     // 3 lanes
  double* P = R + 3 * ld;
  double* G = P + ld;
  double* TMP = G + ld;       // 3 lanes
  double2* WA = reinterpret_cast<double2*>(TMP + 3 * ld + 2);
  WA = reinterpret_cast<double2*>((reinterpret_cast<size_t>(WA) + 15) & ~size_t(15));
  const int wld = c.cy.use_fft ? c.cy.L : 1;
  double2* WB = WA + 2 * wld;
  (void)nx;
  if (PRE) {
    const double* cv = static_cast<const double*>(c.m_cv);
    for (int idx = tid; idx < 3 * ny; idx += nth) {
      int f = idx / ny, k = idx - f * ny;
      CV[f * ld + k] = (i < kx && k < ky) ? cv[((size_t)f * kx + i) * ky + k] : 0.0;
    }
  } else if (i < kx) {
    const double* q = static_cast<const double*>(c.q[0]);
    for (int idx = tid; idx < 3 * ny; idx += nth) {
      int f = idx / ny, k = idx - f * ny;
      TMP[f * ld + k] = q[(size_t)f * kx * ny + (size_t)i * ny + k];
    }
    __syncthreads();
    if (c.cy.use_fft) dct1_fft_r(c.cy, true, TMP, ld, CV, ld, 3, WA, WB, wld, tid, nth);
    else dct1_dense<double>(c.cy, true, TMP, ld, CV, ld, 3, tid, nth);
    for (int idx = tid; idx < 3 * ny; idx += nth) {
      int f = idx / ny, k = idx - f * ny;
      if (k >= ky) CV[f * ld + k] = 0.0;
    }
  } else {
    for (int idx = tid; idx < 3 * ny; idx += nth) CV[(idx / ny) * ld + idx % ny] = 0.0;
  }
  // (Sx f)[i] = diag_i f[i] + low2_{i-2} f[i-2] for composite rows
  void* f3[3] = {c.ux, c.uy, c.temp};
  const BasisDev* xb[3] = {&c.xu, &c.xu, &c.xt};
  for (int idx = tid; idx < 3 * myc; idx += nth) {
    int f = idx / myc, k = idx - f * myc;
    const double* a = static_cast<const double*>(f3[f]);
    const BasisDev& b = *xb[f];
    double v = 0.0;
    bool has = false;
    if (i < mxc) { v = b.unit_diag ? a[(size_t)i * myc + k] : a[(size_t)i * myc + k] * b.diag[i]; has = true; }
    if (i >= 2 && i - 2 < mxc) {
      double t = a[(size_t)(i - 2) * myc + k];
      v = has ? fma(t, b.low2[i - 2], v) : t * b.low2[i - 2];
    }
    SX[f * ld + k] = v;
  }
  const double* p0 = static_cast<const double*>(c.p0);
  for (int k = tid; k < ny; k += nth) P[k] = p0[(size_t)i * ny + k];
  __syncthreads();
  to_ortho<double>(c.ycd, SX, ld, O, ld, 3, tid, nth);
  cheb_diff<double>(c.odd, P, ld, G, ld, ny, 1, 1, TMP, ld, tid, nth);
  const double* gpx = static_cast<const double*>(c.s[0]);
  const double* bco = static_cast<const double*>(c.bc_ortho);
  const double* bcd = static_cast<const double*>(c.bc_diff);
  for (int k = tid; k < ny; k += nth) {
    R[k] = fnms(fnms(O[k], gpx[(size_t)i * ny + k], dt), CV[k], dt);
    double that = O[2 * ld + k] + bco[(size_t)i * ny + k];
    R[ld + k] = fnms(fmas(fnms(O[ld + k], G[k], dt), that, dt), CV[ld + k], dt);
    double ct = CV[2 * ld + k];
    if (CONV == CONV_MIXED && c.m_bclin && i < kx && k < ky) ct = add_bclin(ct, O[ld + k], c.m_bcg, i);
    R[2 * ld + k] = fnms(O[2 * ld + k] + bcd[(size_t)i * ny + k], ct, dt);
  }
  __syncthreads();
  matvec_pinv<double>(c.pinv_y, R, ld, O, ld, 3, tid, nth);
  for (int idx = tid; idx < 3 * myc; idx += nth) {
    int f = idx / myc, k = idx - f * myc;
    static_cast<double*>(c.s[1 + f])[(size_t)i * myc + k] = O[f * ld + k];
  }
}

size_t smem_box_y2(const CaseDev& c) {
  size_t ld = c.ny + 1;
  size_t wld = c.cy.use_fft ? c.cy.L : 1;
  return 17 * ld * 8 + 2 * 2 * wld * 16 + 64;
}

// with the convection term given: no FFT work lanes (box 513^2: three CTAs per SM instead of one)
size_t smem_box_y2_pre(const CaseDev& c) { return 17 * (size_t)(c.ny + 1) * 8 + 64; }

// X2: columns j < myc.  pinv_x then the ADI x solve.  s[1..3] -> s[4..6] (mxc x myc)
// (four CTAs per SM here and in k_box_y3: with 80 registers three fitted; box
// 513 x 513 step 502 -> 475 us, 8 cases of 65 x 65 149 -> 139)
__global__ void __launch_bounds__(256, 4) k_box_x2(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y;
  const int nx = c.nx, myc = c.myc, mxc = c.mxc;
  const int ld = nx + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* IN = reinterpret_cast<double*>(smem);
  double* OUT = IN + 3 * ld;
  double* FAC = OUT + 3 * ld;
  const bool stage = stage_factors(mxc);
  const FdmaDev hu = stage ? stage_fdma_row(c.hu_x, 0, FAC, tid, nth) : c.hu_x;
  const FdmaDev ht = stage ? stage_fdma_row(c.ht_x, 0, FAC + 4 * mxc, tid, nth) : c.ht_x;
  load_lanes3(c.s[1], c.s[2], c.s[3], (size_t)j, myc, nx, IN, ld, tid, nth);
  __syncthreads();
  matvec_pinv<double>(c.pinv_x, IN, ld, OUT, ld, 3, tid, nth);
  fdma_solve2<double>(hu, ht, 2, OUT, ld, 3, 0, 0, tid, nth);
  double* o0 = static_cast<double*>(c.s[4]);
  double* o1 = static_cast<double*>(c.s[5]);
  double* o2 = static_cast<double*>(c.s[6]);
  for (int k = tid; k < mxc; k += nth) {
    const size_t o = (size_t)k * myc + j;
    o0[o] = OUT[k];
    o1[o] = OUT[ld + k];
    o2[o] = OUT[2 * ld + k];
  }
}

size_t smem_box_x2(const CaseDev& c) { return (stage_factors(c.mxc) ? 14 : 6) * (size_t)(c.nx + 1) * 8 + 64; }

// Y3: rows i < mxc.  ADI y solve -> ux*, uy*, temp(new); A = Sy ux*, B = Dy Sy uy*
__global__ void __launch_bounds__(256, 4) k_box_y3(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int i = w.y;
  const int ny = c.ny, myc = c.myc;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* F = reinterpret_cast<double*>(smem);
  double* O = F + 3 * ld;
  double* B = O + 2 * ld;
  double* TMP = B + ld;
  double* FAC = TMP + 2 * ld;
  const bool stage = stage_factors(myc);
  const FdmaDev hu = stage ? stage_fdma_row(c.hu_y, 0, FAC, tid, nth) : c.hu_y;
  const FdmaDev ht = stage ? stage_fdma_row(c.ht_y, 0, FAC + 4 * myc, tid, nth) : c.ht_y;
  load_lanes3(c.s[4], c.s[5], c.s[6], (size_t)i * myc, 1, myc, F, ld, tid, nth);
  __syncthreads();
  fdma_solve2<double>(hu, ht, 2, F, ld, 3, 0, 0, tid, nth);
  to_ortho<double>(c.ycd, F, ld, O, ld, 2, tid, nth);
  cheb_diff<double>(c.odd, O + ld, ld, B, ld, ny, 1, 1, TMP, ld, tid, nth);
  // ux*, uy* -> s[4], s[5] (in place);  temp -> state
  bool bad = false;
  double* us = static_cast<double*>(c.s[4]) + (size_t)i * myc;
  double* vs = static_cast<double*>(c.s[5]) + (size_t)i * myc;
  double* tt = static_cast<double*>(c.temp) + (size_t)i * myc;
  for (int k = tid; k < myc; k += nth) {
    const double u = F[k], v = F[ld + k], t = F[2 * ld + k];
    us[k] = u;
    vs[k] = v;
    tt[k] = t;
    bad |= !(finite_v(u) && finite_v(v) && finite_v(t));
  }
  double* A = static_cast<double*>(c.s[1]);   // mxc x ny
  double* Bs = static_cast<double*>(c.s[2]);  // mxc x ny
  for (int k = tid; k < ny; k += nth) {
    A[(size_t)i * ny + k] = O[k];
    Bs[(size_t)i * ny + k] = B[k];
  }
  if (bad) flag_nonfinite(c.status);
}

size_t smem_box_y3(const CaseDev& c) { return (stage_factors(c.myc) ? 16 : 8) * (size_t)(c.ny + 1) * 8 + 64; }

// X3: columns j < ny.  div = Dx Sx A / s + Sx B  (-> s[3], nx x ny);
// Zf = fwd * pinv_x div  (-> s[1] reused? no: s[6], mxc x ny)
// The eigenbasis product: EIG_DENSE here; EIG_MIXED and EIG_SPLIT as a GEMM that
// follows, from FP32 values (m_z) or from nine-digit lanes (spl_z).
enum { EIG_DENSE = 0, EIG_MIXED = 1, EIG_SPLIT = 2 };
template <int EIG>
__global__ void __launch_bounds__(256) k_box_x3(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y;
  const int nx = c.nx, ny = c.ny, mxc = c.mxc;
  const int ld = nx + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  extern __shared__ double2 smem[];
  double* IN = reinterpret_cast<double*>(smem);  // 2 lanes (mxc)
  double* OR = IN + 2 * ld;                      // 2 lanes (nx)
  double* DV = OR + 2 * ld;                      // div lane
  double* Z = DV + ld;                           // pinv lane
  double* TMP = Z + ld;                          // 2 lanes
  const double* A = static_cast<const double*>(c.s[1]);
  const double* B = static_cast<const double*>(c.s[2]);
  for (int k = tid; k < mxc; k += nth) {
    const double a = __ldcg(A + (size_t)k * ny + j), b = __ldcg(B + (size_t)k * ny + j);
    IN[k] = a;
    IN[ld + k] = b;
  }
  __syncthreads();
  to_ortho<double>(c.xu, IN, ld, OR, ld, 2, tid, nth);
  cheb_diff<double>(c.odd, OR, ld, TMP, ld, nx, 1, 1, TMP + ld, ld, tid, nth);
  double* dv = static_cast<double*>(c.s[3]);
  for (int k = tid; k < nx; k += nth) {
    double v = TMP[k] * inv_asp + OR[ld + k];
    DV[k] = v;
    dv[(size_t)k * ny + j] = v;
  }
  __syncthreads();
  matvec_pinv<double>(c.pinv_x, DV, ld, Z, ld, 1, tid, nth);
  if (EIG == EIG_SPLIT) {
    split_emit9(c.spl_z, j, 1, mxc, c.smat_f.K0, c.smat_f.colex, [&](int, int k) { return Z[k]; },
                reinterpret_cast<int*>(TMP), tid, nth);
    return;
  }
  if (EIG == EIG_MIXED) {
    float* mz = static_cast<float*>(c.m_z);
    for (int r = tid; r < mxc; r += nth) mz[(size_t)r * ny + j] = to_f32(Z[r]);
    return;
  }
  // dense eigenbasis forward along x
  double* zf = static_cast<double*>(c.s[6]);
  for (int r = tid; r < mxc; r += nth) {
    zf[(size_t)r * ny + j] = table_dot<double>(c.pois_fwd + r, mxc, mxc, Z, 1);
  }
}

size_t smem_box_x3(const CaseDev& c) { return 8 * (size_t)(c.nx + 1) * 8 + 64; }

// Y4: rows i < mxc.  pinv_y then the Poisson row solve (eigen row i) -> s[7] (mxc x myc)
// MIX: in FP32 into m_z instead, the input of the eigenbasis GEMM
template <bool MIX>
__global__ void __launch_bounds__(256) k_box_y4(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int i = w.y;
  const int ny = c.ny, myc = c.myc;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* IN = reinterpret_cast<double*>(smem);
  double* OUT = IN + ld;
  const FdmaDev fp = stage_fdma_row(c.pois_y, i, OUT + ld, tid, nth);
  const double* zf = static_cast<const double*>(c.s[6]);
  for (int k = tid; k < ny; k += nth) IN[k] = zf[(size_t)i * ny + k];
  __syncthreads();
  matvec_pinv<double>(c.pinv_y, IN, ld, OUT, ld, 1, tid, nth);
  fdma_solve<double>(fp, OUT, ld, 1, 0, 0, tid, nth);
  if (MIX) {  // FP32 into m_z: the input of the eigenbasis GEMM
    float* wf = static_cast<float*>(c.m_z);
    for (int k = tid; k < myc; k += nth) wf[(size_t)i * myc + k] = to_f32(OUT[k]);
    return;
  }
  double* wv = static_cast<double*>(c.s[7]);
  for (int k = tid; k < myc; k += nth) wv[(size_t)i * myc + k] = OUT[k];
}

size_t smem_box_y4(const CaseDev& c) { return 6 * (size_t)(c.ny + 1) * 8 + 64; }

// column j of the Poisson row solutions (s[7]) as nine-digit lanes
__global__ void __launch_bounds__(256) k_spl_w(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y, myc = c.myc, mxc = c.mxc, tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* W = reinterpret_cast<double*>(smem);
  const double* wv = static_cast<const double*>(c.s[7]);
  for (int k = tid; k < mxc; k += nth) W[k] = wv[(size_t)k * myc + j];
  __syncthreads();
  split_emit9(c.spl_w, j, 1, mxc, c.smat_b.K0, c.smat_b.colex, [&](int, int k) { return W[k]; },
              reinterpret_cast<int*>(W + mxc), tid, nth);
}
static size_t smem_spl_w(const CaseDev& c) { return (size_t)c.mxc * 8 + 64; }

// X4: columns j < myc.  p1 = bwd * W (p1[0][0] = 0).  E = Sx+ Dx Sx^N p1 / s,
// Fv = Sx+ Sx^N p1 (-> s[1], s[2] as mxc x myc), Gp = Sx^N p1 (-> s[0], nx x myc)
// MIX: p1 = bwd * W was computed by a GEMM; read it (and set p1[0][0] = 0).
template <bool MIX>
__global__ void __launch_bounds__(256) k_box_x4(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int j = w.y;
  const int nx = c.nx, myc = c.myc, mxc = c.mxc;
  const int ld = nx + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  const double inv_asp = 1.0 / c.aspect;
  extern __shared__ double2 smem[];
  double* W = reinterpret_cast<double*>(smem);
  double* PV = W + ld;
  double* OR = PV + ld;       // Sx^N p1 (nx)
  double* D = OR + ld;        // 2 lanes: Dx OR / s, OR copy
  double* FO = D + 2 * ld;    // 2 lanes from_ortho
  double* TMP = FO + 2 * ld;  // 2 lanes
  double* p1 = static_cast<double*>(c.p1);
  if (MIX) {
    for (int r = tid; r < mxc; r += nth) {
      double v = p1[(size_t)r * myc + j];
      if (j == 0 && r == 0) {
        v = 0.0;
        p1[0] = 0.0;
      }
      PV[r] = v;
    }
  } else {
    const double* wv = static_cast<const double*>(c.s[7]);
    for (int k = tid; k < mxc; k += nth) W[k] = wv[(size_t)k * myc + j];
    __syncthreads();
    for (int r = tid; r < mxc; r += nth) {
      double acc = table_dot<double>(c.pois_bwd + r, mxc, mxc, W, 1);
      if (j == 0 && r == 0) acc = 0.0;
      PV[r] = acc;
      p1[(size_t)r * myc + j] = acc;
    }
  }
  __syncthreads();
  to_ortho<double>(c.xp, PV, ld, OR, ld, 1, tid, nth);
  cheb_diff<double>(c.odd, OR, ld, TMP, ld, nx, 1, 1, TMP + ld, ld, tid, nth);
  double* gp = static_cast<double*>(c.s[0]);
  for (int k = tid; k < nx; k += nth) {
    D[k] = TMP[k] * inv_asp;
    D[ld + k] = OR[k];
    gp[(size_t)k * myc + j] = OR[k];
  }
  __syncthreads();
  from_ortho<double>(c.xu, D, ld, FO, ld, 2, tid, nth);
  double* e = static_cast<double*>(c.s[1]);
  double* fv = static_cast<double*>(c.s[2]);
  for (int k = tid; k < mxc; k += nth) {
    e[(size_t)k * myc + j] = FO[k];
    fv[(size_t)k * myc + j] = FO[ld + k];
  }
}

size_t smem_box_x4(const CaseDev& c) { return 9 * (size_t)(c.nx + 1) * 8 + 64; }

// Y5: rows i < nx.  ux = ux* - Sy+ Sy^N E ; uy = uy* - Sy+ Dy Sy^N Fv ;
// p0 = (p0 - nu div) + Sy^N Gp / dt
__global__ void __launch_bounds__(256) k_box_y5(const CaseDev* __restrict__ cases, const int4* __restrict__ work) {
  pdl_enter();
  int4 w = work[blockIdx.x];
  const CaseDev& c = cases[w.x];
  if (c.gate != nullptr && c.gate[1] == 0) return;  // case idle this step (serving)
  const int i = w.y;
  const int ny = c.ny, myc = c.myc, mxc = c.mxc;
  const int ld = ny + 1;
  const int tid = threadIdx.x, nth = blockDim.x;
  extern __shared__ double2 smem[];
  double* IN = reinterpret_cast<double*>(smem);  // 3 lanes (myc): E, Fv, Gp
  double* OR = IN + 3 * ld;                      // 3 lanes
  double* D = OR + 3 * ld;                       // 2 lanes: dpdx, dpdy
  double* FO = D + 2 * ld;                       // 2 lanes
  double* TMP = FO + 2 * ld;
  const double* e = static_cast<const double*>(c.s[1]);
  const double* fv = static_cast<const double*>(c.s[2]);
  const double* gp = static_cast<const double*>(c.s[0]);
  if (i < mxc) {
    load_lanes3(e, fv, gp, (size_t)i * myc, 1, myc, IN, ld, tid, nth);
  } else {
    for (int k = tid; k < myc; k += nth) IN[2 * ld + k] = gp[(size_t)i * myc + k];
  }
  __syncthreads();
  if (i < mxc) {
    to_ortho<double>(c.ycn, IN, ld, OR, ld, 2, tid, nth);
    cheb_diff<double>(c.odd, OR + ld, ld, D + ld, ld, ny, 1, 1, TMP, ld, tid, nth);
    for (int k = tid; k < ny; k += nth) D[k] = OR[k];
    __syncthreads();
    from_ortho<double>(c.ycd, D, ld, FO, ld, 2, tid, nth);
    double* ux = static_cast<double*>(c.ux);
    double* uy = static_cast<double*>(c.uy);
    const double* us = static_cast<const double*>(c.s[4]);
    const double* vs = static_cast<const double*>(c.s[5]);
    bool bad = false;
    for (int k = tid; k < myc; k += nth) {
      double a = us[(size_t)i * myc + k] - FO[k];
      double b = vs[(size_t)i * myc + k] - FO[ld + k];
      ux[(size_t)i * myc + k] = a;
      uy[(size_t)i * myc + k] = b;
      bad |= !(finite_v(a) && finite_v(b));
    }
    if (bad) flag_nonfinite(c.status);
  }
  to_ortho<double>(c.ycn, IN + 2 * ld, ld, OR + 2 * ld, ld, 1, tid, nth);
  double* p0 = static_cast<double*>(c.p0);
  const double* dv = static_cast<const double*>(c.s[3]);
  for (int k = tid; k < ny; k += nth) {
    double v = fnms(p0[(size_t)i * ny + k], dv[(size_t)i * ny + k], c.nu);
    p0[(size_t)i * ny + k] = fmas(v, OR[2 * ld + k], c.inv_dt);
  }
}

size_t smem_box_y5(const CaseDev& c) { return 12 * (size_t)(c.ny + 1) * 8 + 64; }

}  // namespace dev

// ---------------------------------------------------------------------------
// host-side launch helpers
// ---------------------------------------------------------------------------
static inline size_t clamp_smem(size_t s) { return (s + 127) & ~size_t(127); }

cudaError_t configure_step_kernels() {
  static PerDeviceFlag done;
  if (done.test()) return cudaSuccess;
  const int big = (int)smem_limit();
  cudaError_t e;
#define SET_ATTR(k)                                                                          \
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, big);             \
  if (e != cudaSuccess) return e;
  SET_ATTR(dev::k_y1<double>);
  SET_ATTR(dev::k_y1<double2>);
  SET_ATTR(dev::k_per_x);
  SET_ATTR((dev::k_per_y2<dev::CONV_Q, 256, 4>));
  SET_ATTR((dev::k_per_y2<dev::CONV_FULL, 256, 1>));
  SET_ATTR((dev::k_per_y2<dev::CONV_FULL, 256, 3>));
  SET_ATTR((dev::k_per_y2<dev::CONV_FULL, 256, 4>));
  SET_ATTR((dev::k_per_y2<dev::CONV_MIXED, 256, 1>));
  SET_ATTR((dev::k_per_y2<dev::CONV_MIXED, 256, 3>));
  SET_ATTR((dev::k_per_y2<dev::CONV_MIXED, 256, 4>));
  SET_ATTR((dev::k_per_y2<dev::CONV_MIXED, 128, 7>));
  SET_ATTR(dev::k_per_y2a);
  SET_ATTR(dev::k_per_y2b);
  SET_ATTR(dev::k_box_x1);
  SET_ATTR(dev::k_box_y2<dev::CONV_Q>);
  SET_ATTR(dev::k_box_y2<dev::CONV_FULL>);
  SET_ATTR(dev::k_box_y2<dev::CONV_MIXED>);
  SET_ATTR(dev::k_box_x2);
  SET_ATTR(dev::k_box_gpx);
  SET_ATTR(dev::k_box_y3);
  SET_ATTR(dev::k_box_x3<dev::EIG_DENSE>);
  SET_ATTR(dev::k_box_x3<dev::EIG_MIXED>);
  SET_ATTR(dev::k_box_x3<dev::EIG_SPLIT>);
  SET_ATTR(dev::k_spl_w);
  SET_ATTR(dev::k_box_y4<false>);
  SET_ATTR(dev::k_box_y4<true>);
  SET_ATTR(dev::k_box_x4<false>);
  SET_ATTR(dev::k_box_x4<true>);
  SET_ATTR(dev::k_box_y5);
#undef SET_ATTR
  e = configure_step_split_kernels();
  if (e != cudaSuccess) return e;
  done.set();
  return cudaSuccess;
}

StepPlan build_step_plan(const CaseDev& c) {
  StepPlan p;
  const bool per = c.kind == KIND_PERIODIC;
  const bool split = c.split != 0 && c.solid_cm == nullptr;
  auto add_if = [&](bool on, int kernel, int lanes, size_t smem) {
    StepLaunch L;
    L.kernel = kernel;
    L.smem = on ? clamp_smem(smem) : 0;
    if (on)
      for (int i = 0; i < lanes; i++) L.items.push_back(make_int4(0, i, 1, 0));
    p.launches.push_back(L);
  };
  auto add = [&](int kernel, int lanes, size_t smem) { add_if(true, kernel, lanes, smem); };
  if (per) {
    add_if(!split, K_Y1_C, c.mxc, dev::smem_y1(c, 1, true));
    add_if(!split, K_PER_X, c.ny, dev::smem_per_x(c));
    add_split_launches(c, split, p);
    // fused Y2 (one CTA per row): faster than the split Y2a/Y2b pair on this
    // GPU because each FP64 warp instruction costs its warp ~64 cycles and the
    // split leaves single-lane CTAs with long per-warp FP64 chains
    add_if(!split, K_PER_Y2, c.mx, dev::smem_per_y2(c));
    add_if(split, K_PER_Y2_CV, c.mx, dev::smem_per_y2_pre(c));
  } else {
    add_if(!split, K_Y1_R, c.mxc, dev::smem_y1(c, 1, false));
    add_if(!split, K_BOX_X1, c.ny, dev::smem_box_x1(c));
    add_split_launches(c, split, p);
    add_if(!split, K_BOX_Y2, c.nx, dev::smem_box_y2(c));
    add_if(split, K_BOX_Y2_CV, c.nx, dev::smem_box_y2_pre(c));
    add(K_BOX_X2, c.myc, dev::smem_box_x2(c));
    add(K_BOX_Y3, c.mxc, dev::smem_box_y3(c));
    const bool eig = split && c.split_eig != 0;
    auto eig_gemm = [&](const SplitLanesDev& s, const SplitMatDev& m, int lanes, void* out, long long es) {
      StepLaunch L;
      L.kernel = K_SPLIT_GEMM;
      L.smem = 0;
      if (eig) L.sjobs.push_back(split_mat_job(s, m, lanes, static_cast<double*>(out), es, c.status));
      p.launches.push_back(L);
    };
    add_if(!eig, K_BOX_X3, c.ny, dev::smem_box_x3(c));
    add_if(eig, K_SPL_X3, c.ny, dev::smem_box_x3(c));
    eig_gemm(c.spl_z, c.smat_f, c.ny, c.s[6], c.ny);
    add(K_BOX_Y4, c.mxc, dev::smem_box_y4(c));
    add_if(eig, K_SPL_W, c.myc, dev::smem_spl_w(c));
    eig_gemm(c.spl_w, c.smat_b, c.myc, c.p1, c.myc);
    add_if(!eig, K_BOX_X4, c.myc, dev::smem_box_x4(c));
    add_if(eig, K_BOX_X4_MIX, c.myc, dev::smem_box_x4(c));
    add(K_BOX_Y5, c.nx, dev::smem_box_y5(c));
  }
  return p;
}

void drop_empty(StepPlan& p) {
  p.launches.erase(
      std::remove_if(p.launches.begin(), p.launches.end(), [](const StepLaunch& L) { return L.empty(); }),
      p.launches.end());
}

// CTAs per SM that k_per_y2's registers have to allow in a launch of so many rows
static int y2_bound(int rows, size_t smem) {
  if (rows <= 2 * kNumSMs) return 1;
  return 3 * (smem + 1024) <= smem_limit() + 1024 ? 4 : 3;  // (1 KB of a CTA's shared memory is the system's)
}
template <int CONV>
static cudaError_t launch_per_y2(int rows, size_t smem, cudaStream_t s, const CaseDev* cases, const int4* work) {
  switch (y2_bound(rows, smem)) {
    case 4: return launch_pdl(dev::k_per_y2<CONV, 256, 4>, rows, 256, smem, s, cases, work);
    case 3: return launch_pdl(dev::k_per_y2<CONV, 256, 3>, rows, 256, smem, s, cases, work);
    default: return launch_pdl(dev::k_per_y2<CONV, 256, 1>, rows, 256, smem, s, cases, work);
  }
}

cudaError_t launch_step_kernel(int kernel, int nblocks, size_t smem, cudaStream_t s, const CaseDev* cases,
                               const int4* work) {
  dim3 g(nblocks), b(256);
  switch (kernel) {
    case K_Y1_C: return launch_pdl(dev::k_y1<double2>, g, b, smem, s, cases, work);
    case K_Y1_R: return launch_pdl(dev::k_y1<double>, g, b, smem, s, cases, work);
    case K_PER_X: return launch_pdl(dev::k_per_x, g, b, smem, s, cases, work);
    case K_PER_Y2: return launch_pdl(dev::k_per_y2<dev::CONV_Q, 256, 4>, g, b, smem, s, cases, work);
    case K_PER_Y2_PRE: return launch_per_y2<dev::CONV_MIXED>(nblocks, smem, s, cases, work);
    case K_PER_Y2A: return launch_pdl(dev::k_per_y2a, g, b, smem, s, cases, work);
    case K_PER_Y2B: return launch_pdl(dev::k_per_y2b, g, b, smem, s, cases, work);
    case K_BOX_X1: return launch_pdl(dev::k_box_x1, g, b, smem, s, cases, work);
    case K_BOX_Y2: return launch_pdl(dev::k_box_y2<dev::CONV_Q>, g, b, smem, s, cases, work);
    case K_BOX_Y2_PRE: return launch_pdl(dev::k_box_y2<dev::CONV_MIXED>, g, b, smem, s, cases, work);
    case K_PER_Y2_CV: return launch_per_y2<dev::CONV_FULL>(nblocks, smem, s, cases, work);
    case K_BOX_Y2_CV: return launch_pdl(dev::k_box_y2<dev::CONV_FULL>, g, b, smem, s, cases, work);
    case K_SPL_X3: return launch_pdl(dev::k_box_x3<dev::EIG_SPLIT>, g, b, smem, s, cases, work);
    case K_SPL_W: return launch_pdl(dev::k_spl_w, g, b, smem, s, cases, work);
    case K_BOX_X2: return launch_pdl(dev::k_box_x2, g, b, smem, s, cases, work);
    case K_BOX_GPX: return launch_pdl(dev::k_box_gpx, g, b, smem, s, cases, work);
    case K_BOX_Y3: return launch_pdl(dev::k_box_y3, g, b, smem, s, cases, work);
    case K_BOX_X3: return launch_pdl(dev::k_box_x3<dev::EIG_DENSE>, g, b, smem, s, cases, work);
    case K_BOX_X3_MIX: return launch_pdl(dev::k_box_x3<dev::EIG_MIXED>, g, b, smem, s, cases, work);
    case K_BOX_Y4: return launch_pdl(dev::k_box_y4<false>, g, b, smem, s, cases, work);
    case K_BOX_Y4_MIX: return launch_pdl(dev::k_box_y4<true>, g, b, smem, s, cases, work);
    case K_BOX_X4: return launch_pdl(dev::k_box_x4<false>, g, b, smem, s, cases, work);
    case K_BOX_X4_MIX: return launch_pdl(dev::k_box_x4<true>, g, b, smem, s, cases, work);
    case K_BOX_Y5: return launch_pdl(dev::k_box_y5, g, b, smem, s, cases, work);
    case K_PER_Y2_PRE_T128: return launch_pdl(dev::k_per_y2<dev::CONV_MIXED, 128, 7>, g, dim3(128), smem, s, cases, work);
    case K_BOX_Y2_PRE_T128: return launch_pdl(dev::k_box_y2<dev::CONV_MIXED>, g, dim3(128), smem, s, cases, work);
    case K_BOX_X3_MIX_T128: return launch_pdl(dev::k_box_x3<dev::EIG_MIXED>, g, dim3(128), smem, s, cases, work);
    case K_BOX_Y5_T128: return launch_pdl(dev::k_box_y5, g, dim3(128), smem, s, cases, work);
    case K_SPL_Y1_R: case K_SPL_Y1_C: case K_SPL_X1_BOX: case K_SPL_X1_PER: case K_SPL_PROD: case K_SPL_Q:
      return launch_step_split_kernel(kernel, nblocks, smem, s, cases, work);
    default: return launch_mixed_kernel(kernel, nblocks, smem, s, cases, work);
  }
}

}  // namespace rbc
