// rb_kernels.cuh -- launch-parameter structs and kernel entry points shared between the
// CUDA translation units and the host-side C ABI (rb_api.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace rb {

// Real-valued BLAS1 reductions (one binned accumulator per result)
enum Op1 : int {
  kOpSum = 0,   // sum x_i                       (dmdsum / smssum)
  kOpDot = 1,   // sum fl(x_i * y_i)             (dmddot / smsdot)
  kOpSsq = 2,   // sum fl((x_i * (1/scl))^2)     (dmdssq), running power-of-two scale
  kOpAsum = 3,  // sum |x_i|                     (dmdasum / smsasum)
};
// Complex BLAS1 reductions (two accumulators, real and imaginary)
enum OpC : int {
  kOpCSum = 0,   // sum x_i                      (zmzsum / cmcsum)
  kOpCDotc = 1,  // sum conj(x_i) * y_i          (zmzdotc / cmcdotc)
  kOpCDotu = 2,  // sum x_i * y_i                (zmzdotu / cmcdotu)
};

// Workspace used by a grid-wide reduction: one partial record per CTA plus an arrival
// ticket. The last CTA to arrive merges the records and resets the ticket to zero.
struct GridScratch {
  void* records;       // >= gridDim.x * record_bytes
  unsigned* ticket;    // zero on entry, zero again on exit
  size_t bytes;        // capacity of `records`
};

struct Blas1Args {
  long long n;               // number of elements
  const void* x;             // device pointer
  long long incx;            // stride in elements (>= 0)
  const void* y;             // device pointer (dot only)
  long long incy;
  long long head;            // vector path: elements before the aligned body
  long long body_end;        // vector path: end of the body of whole warp tiles
  GridScratch scratch;
  void* acc;                 // device binned accumulator (reference layout), read then written
  double* scale;             // ssq: device scale, read then written (may be null: 0)
  void* result;              // device converted result (T, or 2 T for complex); may be null
  int sqrt_result;           // ssq: write scale*sqrt(conv) instead of conv
  int fold;                  // the fold (read by the run-time fold kernels)
};

// Launch helpers implemented in rb_blas1.cu; return cudaSuccess or the launch error.
// `vec` selects the 16-byte vector body (contiguous, aligned inputs).
cudaError_t launch_blas1_d(int fold, int op, bool vec, int grid, int block,
                           const Blas1Args& a, cudaStream_t s);
cudaError_t launch_blas1_s(int fold, int op, bool vec, int grid, int block,
                           const Blas1Args& a, cudaStream_t s);
cudaError_t launch_blas1_z(int fold, int op, bool vec, int grid, int block, const Blas1Args& a,
                           cudaStream_t s);
cudaError_t launch_blas1_c(int fold, int op, bool vec, int grid, int block, const Blas1Args& a,
                           cudaStream_t s);

// Complex elements per warp tile of the complex kernels' vector body, for complex elements
// of `elem` bytes (8 or 16): 32 lanes x 4 (sum) or 2 (dotc) 16-byte vectors.
__host__ __device__ constexpr int blas1_complex_tile(size_t elem, int op) {
  return 32 * (op == kOpCSum ? 4 : 2) * (int)(16 / elem);
}

// out (device double_binned) += each of `count` device double_binned states.
cudaError_t launch_merge_states(int fold, int count, const double* states, double* out,
                                cudaStream_t s);

// Bytes of one per-CTA record for the given element size, fold and component count.
inline size_t blas1_record_bytes(size_t elem, int fold, int comps) {
  // per component: fold primaries, fold carries, flags word, scale (ssq)
  size_t per = (2 * (size_t)fold + 2) * elem;
  if (per < 16) per = 16;
  return ((comps * per) + 15) / 16 * 16 + 16;
}

// Launchers of one fold (instantiated in rb_blas1_f<F>.cu)
struct Blas1FoldOps {
  cudaError_t (*real_d)(int op, bool vec, int grid, int block, const Blas1Args& a, cudaStream_t s);
  cudaError_t (*real_s)(int op, bool vec, int grid, int block, const Blas1Args& a, cudaStream_t s);
  cudaError_t (*cplx_z)(int op, bool vec, int grid, int block, const Blas1Args& a, cudaStream_t s);
  cudaError_t (*cplx_c)(int op, bool vec, int grid, int block, const Blas1Args& a, cudaStream_t s);
  cudaError_t (*merge)(int count, const double* states, double* out, cudaStream_t s);
  const void* (*kernel)(char type, int op, bool vec);
};
extern const Blas1FoldOps blas1_fold2, blas1_fold3, blas1_fold4, blas1_fold5, blas1_fold6,
    blas1_fold7, blas1_fold8;

// ---- BLAS2/3 ------------------------------------------------------------------------
enum OutMode : int {
  kOutValue = 0,    // reproBLAS_r*: init from beta*y (values), write converted values
  kOutBinned = 1,   // binnedBLAS_dbd*: merge into the caller's binned states
};

// Failure-path test hook (rb_runtime.cu): stop_after / wait_polls for the next TMA-fed
// kernels (stop_after < 0 and wait_polls 0 when unset).
void pipeline_fault(long long* stop_after, long long* wait_polls);

// One gemm of any element type. E is the real element type; complex operands are interleaved
// (re, im) pairs and every stride counts whole (complex) elements.
template <typename E>
struct XGemmArgs {
  long long M, N, K;
  const E* A;
  long long sai, sak;         // op(A)_ik = A[i*sai + k*sak]
  const E* B;
  long long sbk, sbj;         // op(B)_kj = B[k*sbk + j*sbj]
  E ar, ai, br, bi;
  int alpha_one;
  int conja, conjb;           // conjugate op(A) / op(B) (complex ConjTrans)
  int mode;
  E* C;                       // kOutValue
  E* Cbin;                    // kOutBinned
  long long sci, scj;         // C_ij at offset i*sci + j*scj (values or states)
};

// Decomposition of one gemm (rb_gemm_tile.cuh). Work is counted in units: one K block of one
// C tile. The units, tile-major, are split evenly over `grid` CTAs; a tile cut between CTAs
// leaves one partial state per CTA in `scratch` and is finished by the last of them to
// arrive (`tickets`, one per tile, zero on entry and on exit).
struct GemmPlan {
  long long units;            // tiles * nkb
  long long nkb;              // K blocks per tile
  long long ntn;              // tiles along N
  long long tiles;
  int grid;
  int cut;                    // some tile is cut: scratch and tickets are needed
  int shape;                  // kernel variant (tile shape)
  size_t scratch_bytes;
  void* scratch;
  unsigned* tickets;
};

// One gemv of any element type (rb_gemv_stream.cuh): A is the stored matrix seen row-major.
template <typename E>
struct XGemvArgs {
  long long R, C;             // A is R x C; the rows kernel has R outputs, the columns kernel C
  const E* A;
  long long lda;
  const E* x;
  long long incx;
  E ar, ai, br, bi;           // alpha, beta (imaginary parts 0 for real elements)
  int alpha_one;              // skip the alpha multiply
  int conj;                   // conjugate A's elements (complex ConjTrans)
  int mode;                   // kOutValue / kOutBinned
  int phases;                 // phases the rows of A are taken in (1, 2, 4; rb_gemv_stream.cuh)
  E* y;                       // kOutValue: values (stride incy)
  E* ybin;                    // kOutBinned: binned states (stride incy states)
  long long incy;
  // decomposition into stages (rb_gemv_stream.cuh)
  int nb;                     // stages per unit
  int q, rem, parts;          // split over the CTAs (Split)
  E* scratch;                 // partial states of units cut between CTAs
  unsigned* tickets;          // of cut units, zero on entry and on exit (null: a second kernel sums)
  int* status;                // set to 2 when a pipeline wait gives up
  int groups;                 // thread groups per output (2, 4, 8)
  // failure-path test hook (rb_debug_pipeline_fault): each CTA's copy warp issues at most
  // `stop_after` stages (< 0: all), and consumers give up waiting for a stage's data after
  // `wait_polls` polls (0: the default ~2 s)
  long long stop_after;
  long long wait_polls;
};

// One tensor map of A per phase.
struct GemvMaps {
  CUtensorMap m[4];
};

template <typename E>
struct XOps {
  // whether gemv takes maps (the streaming kernel of rows or columns) on the current device
  cudaError_t (*gemv_streams)(bool rows, bool* can);
  // maps == nullptr: the direct kernels (g.groups, g.parts: their split of a reduction)
  cudaError_t (*gemv)(const XGemvArgs<E>& g, const GemvMaps* maps, bool rows, int grid, cudaStream_t s);
  // decomposition of an M x N x K product (whole_tiles: no tile is cut between CTAs)
  cudaError_t (*gemm_plan)(long long M, long long N, long long K, int sms, bool whole_tiles,
                           GemmPlan* p);
  cudaError_t (*gemm)(const XGemmArgs<E>& g, const GemmPlan& p, cudaStream_t s);
};
// Kernels of folds 2..8, per element type (rb_blas23_[dszc]{2_4,5_8}.cu).
extern const XOps<double> xops_d_f2, xops_d_f3, xops_d_f4, xops_d_f5, xops_d_f6, xops_d_f7, xops_d_f8;
extern const XOps<float> xops_s_f2, xops_s_f3, xops_s_f4, xops_s_f5, xops_s_f6, xops_s_f7, xops_s_f8;
extern const XOps<double> xops_z_f2, xops_z_f3, xops_z_f4, xops_z_f5, xops_z_f6, xops_z_f7, xops_z_f8;
extern const XOps<float> xops_c_f2, xops_c_f3, xops_c_f4, xops_c_f5, xops_c_f6, xops_c_f7, xops_c_f8;

bool fold_supported(int fold);
// Folds of the register-resident kernels (2..kMaxFold, a template parameter) and the largest
// folds the reference accepts, binned_DBMAXFOLD and binned_SBMAXFOLD (include/binned.h:123,
// 131), served above kMaxFold by the run-time fold kernels of rb_foldn.cu.
constexpr int kMaxFold = 8;
constexpr int kMaxFoldD = 52;
constexpr int kMaxFoldS = 21;
// largest fold for elements of real type 'd' / 'z' (FP64) or 's' / 'c' (FP32)
inline int max_fold(char type) { return (type == 'd' || type == 'z') ? kMaxFoldD : kMaxFoldS; }

// ---- run-time fold kernels (rb_foldn.cu) -------------------------------------------------
extern const Blas1FoldOps blas1_fold_n;   // reads the fold from Blas1Args::fold
// merge `count` packed states of kind 'd', 's', 'z', 'c' (sq: [scale, state] records)
cudaError_t merge_states_n(char kind, bool sq, int fold, int count, const void* states,
                           void* out, cudaStream_t s);

}  // namespace rb
