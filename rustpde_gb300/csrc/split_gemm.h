// split_gemm.h -- dense operators applied along FP64 lanes on the tensor cores
// without losing precision.
//
// This GPU issues two FP64 operations per clock and SM; its bf16 tensor cores
// multiply about 1600 times as fast.  A dense transform of FP64 lanes is
// therefore computed from exact integer digits (the error-free splitting of
// Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication", Numer. Algorithms 59, 2012): every lane is scaled by its
// largest exponent to 56-bit integers, every operator to 55-bit ones, both cut
// into seven balanced base-256 digits.  A digit is exact in bf16, a product of
// two in FP32, and so are the sums of products in the tensor-core accumulators
// (integers below 2^24; see split_gemm.cu).  Digit pairs of equal weight share
// an accumulator; the pairs that matter to FP64 precision are the 34 with
// i + j <= 7.  The epilogue adds the eight accumulators in 64-bit integers and
// rounds once to FP64: nothing runs on the FP64 pipe.
//
// The parity of the Chebyshev nodes (and of sines and cosines) halves the
// products: an operator is two lists of terms, E and O, that see only the even
// and odd parts of a lane (see SplitJobDev).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

namespace rbc {

constexpr int kSplitLanes = 128;      // lanes per tile (tcgen05 M)
constexpr int kSplitDigits = 7;
constexpr int kSplitK = 16;           // terms per chunk (one bf16 MMA k-step)
constexpr int kSplitTile = 32;        // outputs per tile (16 in a short last one)
constexpr int kNumSMs = 152;  // of the GB300
constexpr int kSplitNarrowTiles = kNumSMs;  // launches of at most so many wide tiles take narrow ones
constexpr int kSplitChunkBytes = kSplitDigits * kSplitLanes * kSplitK * 2;  // digits of 128 lanes x 16 terms
// A lane's value with significand m (53 bits) and biased exponent ef becomes the
// integer (m << shl) >> (emax - ef), emax the lane's largest exponent: below
// 2^55 with shl = 2, and with shl = 1 where a term is the sum of two values.
constexpr int kSplitShlValue = 2, kSplitShlSum = 1;
constexpr int kSplitOpBits = 54;      // operator integers: w 2^kSplitOpBits, |w| <= 1

// Digit buffer of a set of lanes: for every block of 128 lanes the chunks of
// list E, then those of list O; a chunk holds its seven digit planes, each in
// the K-major core-matrix order of the tensor core (8 lanes x 16 bytes).
struct SplitLanesDev {
  unsigned char* dig;
  int* ex;     // per lane: biased exponent of the lane's largest term (0x7ff: not finite)
  int cE, cO;  // chunks of the two lists
};
inline int split_chunks(int k) { return (k + kSplitK - 1) / kSplitK; }
size_t split_dig_bytes(int lanes, int cE, int cO, int digits = kSplitDigits);

// out[n] (lane l) of one lane set.  Two lists (nc[1] > 0): values E_n + O_n,
// and E_n - O_n at output mirror - n for m_lo <= n < m_hi.  One list: that
// list's sum.  Lane l = (q * parts + p) * nf + f stores output n at
// out[f fs + q qs + p ps + n es].
struct SplitJobDev {
  const unsigned char* dig;
  const int* ex;
  const unsigned char* w;    // packed operator (SplitOp), 32-wide tiles
  const unsigned char* w16;  // the same in 16-wide tiles
  double* out;
  unsigned int* status;    // receives kStatusGemmTimeout, or null (a lost tile's outputs become NaN either way)
  const int* active;       // when set and 0, the job's tiles do nothing (serving gate)
  long long fs, qs, ps, es;
  int lanes, nf, parts;
  int ctot;                // chunks per lane block in dig
  int c0[2], nc[2];        // first chunk and count of each list
  int N;
  int ex_bias;             // a sum's unit is 2^(ex + ex_bias)
  int mirror, m_lo, m_hi;
  int digits;              // 7, or 9 (one sum over both lists)
  const int* rowex;        // 9 digits: per output, a power of two
};

// Packed operator rows: tile by tile (kSplitTile outputs, a last one of 16
// when 16 or fewer are left; and all of 16), chunk by chunk, digit planes side
// by side.
struct SplitOp {
  int N = 0, K[2] = {0, 0};
  std::vector<unsigned char> bytes, bytes16;
};
// E and O: row-major N x K[list] integers (|.| <= 2^kSplitOpBits)
SplitOp pack_split_op(const std::vector<int64_t>& E, int KE, const std::vector<int64_t>& O, int KO, int N);

// A general n x n matrix in nine digits: entry (r, k) is w 2^(colex[k] + rowex[r]),
// |w| < 1 and w in 70 bits.  Terms are x_k 2^colex[k] in 71 bits (split_emit9):
// a product keeps what FP64 would at any ratio of the terms up to 2^17.  The
// terms are two lists (an accumulator's sums stay below 2^24), added at the end.
constexpr int kSplitShl9 = 18, kSplitOpBits9 = 70;
constexpr int kSplitBadLane9 = 0x7fffff;  // a lane's exponent when it is not finite
inline int split_ex_bias9() { return 56 - 1075 - kSplitShl9 - kSplitOpBits9; }
struct SplitMat {
  int N = 0, K[2] = {0, 0};
  std::vector<int> colex, rowex;
  std::vector<unsigned char> bytes16;
};
SplitMat pack_split_mat(const std::vector<double>& M, int n);

// The barrier (of two) and the phase parity that say a list's accumulators are
// complete.  A barrier per list, because nothing holds the MMA thread back
// between the lists where each has columns of its own: on one barrier it could
// complete both lists' phases before a warp has looked once, and a wait for the
// first phase's parity then never ends (a try_wait sees only whether the
// barrier is past the phase in hand).
struct SplitAccWait {
  int barrier;
  uint32_t parity;
};
__host__ __device__ constexpr SplitAccWait split_acc_wait(int list) { return {list, 0}; }

// Whether an MMA thread that gave up after `issued` of `total` chunks commits
// once more, so that the tile can wait for what it issued: the last chunks free
// no buffer and so commit nothing before their list's end.
__host__ __device__ constexpr bool split_drain_commit(int issued, int total) { return issued > 0 && issued < total; }

// tiles (job, first lane, first output, tile width)
void split_tiles(const std::vector<SplitJobDev>& jobs, std::vector<int4>& tiles);
cudaError_t configure_split_kernels();
cudaError_t launch_split_gemm(const SplitJobDev* jobs, const int4* tiles, int ntiles, int digits, cudaStream_t st);
// at most two jobs, passed by value (no tables)
cudaError_t launch_split_gemm_one(const SplitJobDev* jobs, int njobs, cudaStream_t st);
cudaError_t set_split_wait_limit(long long polls);  // as set_gemm_wait_limit

// Unit exponent of a job's sums (SplitJobDev::ex_bias): terms with shift shl,
// operator integers w 2^(kSplitOpBits + wshift).  The kernel's sums are in
// units of 2^56 products.
inline int split_ex_bias(int shl, int wshift) { return 56 - 1075 - shl - kSplitOpBits - wshift; }

}  // namespace rbc
