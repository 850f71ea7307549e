// step_split.h -- the FP64 step's transforms on the tensor cores (step_split.cu).
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "rbc_dev.h"
#include "split_gemm.h"

namespace rbc {

struct StepPlan;
class Arena;

// Split operators (host form) of the Chebyshev and Fourier transforms.
enum SplitOpKind {
  SOP_CHEB_BWD = 0,  // two lists: values j, n-1-j from the even and odd coefficients
  SOP_CHEB_FWD_E,    // one list: even coefficients (rows) from v_j + v_{n-1-j}
  SOP_CHEB_FWD_O,    //           odd coefficients from v_j - v_{n-1-j}
  SOP_C2R,           // two lists: values j, n-j from the real and the imaginary parts
  SOP_R2C_RE,        // one list: real parts from v_j + v_{n-j}
  SOP_R2C_IM         //           imaginary parts from v_j - v_{n-j}
};
// terms of the two lists of a transform of length n (the E list's, the O list's)
void split_terms(bool fourier, int n, int K[2]);
// rows: outputs to keep (one-list kinds; all for the others).  wshift: see split_ex_bias.
SplitOp make_split_op(int kind, int n, int rows, int* wshift);

// The same on the current device, shared by everything of the size (shared_dev.h); owner: the
// user's arena.
SplitOpDev shared_split_op(Arena& owner, int kind, int n, int rows);
SplitMatDev shared_split_mat(Arena& owner, int kind, int n, bool poisson, bool fwd);

// Whether a case of this size runs its FP64 transforms as split GEMMs.
bool split_step_size(const CaseDev& c);
// The launches up to the convection term m_cv (S1, GEMM, S2, GEMM, S3, GEMM, S4, GEMM)
// (on = false: the same launches without work)
void add_split_launches(const CaseDev& c, bool on, StepPlan& p);
// out[l ls + n es] = the two lists of a transform applied to lane l
SplitJobDev split_op_job(const SplitLanesDev& s, const SplitOpDev& op, int lanes, int shl, double* out, long long ls,
                         long long es, unsigned int* status);
// out[r es + lane] = the matrix applied to nine-digit lanes
SplitJobDev split_mat_job(const SplitLanesDev& s, const SplitMatDev& m, int lanes, double* out, long long es,
                          unsigned int* status);
// Whether a box of this size also runs its Poisson eigenbasis products so.
bool split_eig_size(const CaseDev& c);
cudaError_t configure_step_split_kernels();
cudaError_t launch_step_split_kernel(int kernel, int nblocks, size_t smem, cudaStream_t s, const CaseDev* cases,
                                     const int4* work);

}  // namespace rbc
