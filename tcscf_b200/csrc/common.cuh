// Shared declarations of libtcscf_gpu.so: the context, device-resident grids and tensors, error
// plumbing and small device helpers.  Everything here is product code for sm_100a.
#pragma once

#include <cuda_runtime.h>
#include <cublas_v2.h>
#include <cusolverDn.h>
#include <nvtx3/nvToolsExt.h>
#include <cmath>
#include <cstdint>
#include <array>
#include <map>
#include <string>
#include <vector>

#include "../../include/tcscf_gpu.h"
#include "basis.cuh"

namespace tcscf {

constexpr int kMaxL = 12;            // highest angular momentum the device basis evaluator accepts
constexpr double kPi = 3.141592653589793238462643383279502884;

// Per basis function data the device evaluators read (SlaterTypeOrbital.hpp:27-37 fields plus the
// real-harmonic type used by the tensor paths).


struct Grid {
  int64_t n = 0;
  int ndim = 3;
  double * pts = nullptr;   // [3][n] Cartesian (y row zero for 2-D grids)
  double * w = nullptr;     // [n]
  // basis
  int nb = 0;
  int hasGrad = 0;
  std::vector<tcscf_sto> basis;
  DevSto * dsto = nullptr;  // [nb]
  double * phiR = nullptr;  // real-harmonic basis values [n][nb]
  double * vals = nullptr;  // reference-basis values [n][nb] (complex for ndim 3, real for ndim 2)
  double * grads = nullptr; // [n][nb][3] complex
  // tensor-path cache of the transposed, BF16-split weighted basis values (depends only on the
  // grid and basis, so it is packed once per grid)
  void * vtCache = nullptr;
  int vtNB = 0;
  int64_t vtN2pad = 0;
  double vtScale = 0;
};

// A kept Fji / Vji tensor.  The r12 kernels are real and each element integrates a product of two basis functions, so in the
// real-harmonic basis the tensor is real and symmetric: it is kept as planes [n1][1 or 3][plane] of nb rows
// tensorStride(nb) doubles apart, half the complex [nb][nb](3) layout of the reference basis (a 2-D r2 grid's real Fji: the
// same), which tensorToReference forms where a routine or the host wants it
struct Tensor {
  double * d = nullptr;
  int64_t n1 = 0;
  int nb = 0;
  int isComplex = 1;   // of the reference layout (0: a 2-D r2 grid's real Fji)
  int vec = 0;         // 3 components (Vji)
};
// Row stride of a plane, and doubles per plane.  Up to kTensorPadNb functions, where the fused transcorrelated build copies planes
// as they are, rows are padded to a multiple of 4 and planes to 4 (mod 8), zeros behind and below: the fragments of 8 planes
// then lie on different shared-memory banks and every plane on a 16-byte boundary (24 functions 580 doubles for 576, 7 functions 68 for 49)
constexpr int kTensorPadNb = 32;
__host__ __device__ constexpr int tensorStride(int nb) { return nb > kTensorPadNb ? nb : (nb + 3) / 4 * 4; }
__host__ __device__ constexpr int tensorPlane(int nb) { return tensorStride(nb) * tensorStride(nb) + (nb > kTensorPadNb ? 0 : 4); }

// what the context's pool keeps of released memory
constexpr uint64_t kPoolKeepBytes = uint64_t(4) << 30;

struct Scratch {
  void * p = nullptr;
  size_t bytes = 0;
};

// pairs (r1 index, r2 index) of two grids that the tensor-core kernels drop for FP32 resolution but
// that are not exactly coincident in FP64 (near_pairs.cu); d is device memory, null when count is 0
struct NearList {
  int2 * d = nullptr;
  int count = 0;
};

}  // namespace tcscf

struct tcscf_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cusolverDnHandle_t solver = nullptr;
  cublasHandle_t blas = nullptr;   // created on first use (4- and 6-index tensors)
  // stream-ordered pool of the grid buffers (points, weights, basis values and gradients, the
  // packed tensor-path operand) and kept tensors: grids and tensors created and destroyed between SCF runs reuse its memory
  // without driver allocations or the device-wide synchronisation of cudaFree
  cudaMemPool_t gridPool = nullptr;
  std::string err;
  std::map<int, tcscf::Grid> grids;
  std::map<int, tcscf::Tensor> tensors;
  int nextId = 1;
  // ev[0] / ev[1] bracket a whole call; ev[2 + 2 k] / ev[3 + 2 k] the k-th contraction of a Fock build (up to two
  // spins, real and imaginary parts), read after the call's last synchronisation
  cudaEvent_t ev[10] = {};
  int evPart = 0;
  cudaEvent_t evStart() const { return ev[2 + 2 * evPart]; }
  cudaEvent_t evStop() const { return ev[3 + 2 * evPart]; }
  double lastContractionMs = 0, lastTotalMs = 0;
  int lastLaunches = 0;
  int launchCount = 0;
  int diisSize = 0;   // Pulay DIIS history length of tcscf_scf (0: plain Roothaan iterations)
  // CUDA graph of the most recent batched tensor launch sequence and the launch parameters it was
  // captured with (replayed while a batch repeats them); capture / replay counts
  cudaGraphExec_t tensorGraph = nullptr;
  std::vector<uint64_t> tensorGraphKey;
  int graphCaptures = 0, graphReplays = 0;
  int realEigen = 0;  // tcscf_scf solves a Fock matrix that is real in the real-harmonic basis there
  // set while a conditional graph body is captured: the contraction routines then record no timing
  // events (event nodes are not allowed inside a conditional body)
  int capturing = 0;
  // autotuner (tcscf_set_autotune): the measured schedule (r2 split count, tile class) of the tensor-path launch per shape
  // {n1, n2, padded nb, padded rank, precision}, the split policy per batch signature, the policy
  // the batch build applies (1: the default rule, 0: no split, k > 1: k x the default split),
  // candidate measurements taken, and the two events that time them
  int autotune = 0;
  std::map<std::vector<int64_t>, std::array<int, 3>> tunedSplit;   // {r2 split, T tile width, TMA stages}
  std::map<std::vector<int64_t>, int> tunedBatchPolicy;
  int batchSplitPolicy = 1;
  int tuneMeasurements = 0;
  cudaEvent_t tuneEv[2] = {nullptr, nullptr};
  std::map<std::string, tcscf::Scratch> scratch;
  // near-coincident pair lists per (r1 grid, r2 grid), found on the first tensor-core use of the pair
  std::map<std::pair<const void *, const void *>, tcscf::NearList> nearPairs;
  // device buffers of the most recent direct Fock build (for tcscf_last_potentials)
  const double * lastVH = nullptr;
  const double * lastT = nullptr;
  int64_t lastN1 = 0;
  int lastNb = 0;
};

namespace tcscf {

int fail(tcscf_ctx * ctx, int code, std::string const & msg);

#define TCSCF_CUDA(ctx, call)                                                                 \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return ::tcscf::fail((ctx), TCSCF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

#define TCSCF_LAUNCH(ctx)                                                                     \
  do {                                                                                        \
    (ctx)->launchCount++;                                                                     \
    cudaError_t e_ = cudaGetLastError();                                                      \
    if (e_ != cudaSuccess)                                                                    \
      return ::tcscf::fail((ctx), TCSCF_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e_)); \
  } while (0)

#define TCSCF_CHECK(ctx, cond, code, msg)                                                     \
  do {                                                                                        \
    if (!(cond)) return ::tcscf::fail((ctx), (code), (msg));                                  \
  } while (0)

#define TCSCF_TRY(expr)                                                                       \
  do {                                                                                        \
    int s_ = (expr);                                                                          \
    if (s_ != TCSCF_OK) return s_;                                                            \
  } while (0)

// NVTX range named after the enclosing C-ABI function: profilers that record NVTX show each call
// (and filter kernels by it); without such a tool attached the push and pop do nothing
struct NvtxRange {
  explicit NvtxRange(char const * name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(NvtxRange const &) = delete;
  NvtxRange & operator=(NvtxRange const &) = delete;
};
#define TCSCF_NVTX() ::tcscf::NvtxRange tcscfNvtxRange_(__func__)

// context-owned scratch buffer, grown on demand and kept until the context is destroyed
int scratch(tcscf_ctx * ctx, char const * name, size_t bytes, void ** out);

Grid * findGrid(tcscf_ctx * ctx, int id);

// grid buffers from the context's pool, ordered on ctx->stream; every allocation is checked to be
// 256-byte aligned (vector loads and TMA descriptors rely on it)
int gridAllocBytes(tcscf_ctx * ctx, void ** p, size_t bytes);
template <class T> int gridAlloc(tcscf_ctx * ctx, T ** p, size_t bytes)
{
  void * q = nullptr;
  int const st = gridAllocBytes(ctx, &q, bytes);
  *p = static_cast<T *>(q);
  return st;
}
// returns a grid buffer to the pool in stream order (null is ignored)
void gridRelease(tcscf_ctx * ctx, void * p);
// releases every buffer of a grid and clears its pointers
void gridReleaseAll(tcscf_ctx * ctx, Grid & g);

inline unsigned gridBlocks(int64_t n, int threads)
{
  int64_t b = (n + threads - 1) / threads;
  return unsigned(b < 1 ? 1 : (b > 1048576 ? 1048576 : b));
}

// U coefficient U[k][i] of the unitary complex -> real-harmonic map phiR_k = sum_i U[k][i] phi_i (i = k or its partner)
__device__ __forceinline__ double2 uRow(const DevSto * s, int k, int i)
{
  double const h = 0.70710678118654752440;
  int const t = s[k].rtype;
  if (i == k) return t == 0 ? make_double2(1, 0) : (t == 1 ? make_double2(h, 0) : make_double2(0, h));
  return t == 1 ? make_double2(h, 0) : make_double2(0, -h);
}

// ---- kernels shared between translation units -------------------------------------------------
// r12 kernel evaluation in FP64 (scalar kernels); returns 0 for an exactly coincident pair.
struct OchiDev {
  double a, a12;
  int nterms;
  int S[8][3];
  double c[8][2];
};

// 1/r12 from a finite r12^2 >= 0, 0 for an exactly coincident pair.  The hardware estimate y (rsqrt.approx.ftz.f64 works
// on the high word: no conversions) is refined by the binomial series of (1 - e)^(-1/2) to
// second order, y + y e (1/2 + 3/8 e) with e = 1 - x y^2 (Householder's third-order step), so one step of five FP64 operations
// does what two quadratic Newton steps (seven) do: within 1.24 x 2^-53 over all exponents (tests/test_gpu_inv_r12.py), the
// rounding of the step itself (1.5 at most), so the series' next term is below the last place.  The estimate of zero, and of the subnormal
// numbers the instruction takes for zero (points closer than 2^-511), is cleared on the ALU by the high word, which leaves the FP64 pipe alone.
__device__ __forceinline__ double invR12(double r2)
{
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
  y = __hiloint2double(__double2hiint(r2) < 0x00100000 ? 0 : __double2hiint(y), 0);
  double const e = fma(-r2 * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// D += A B on the FP64 tensor cores: A[r][k] at lane 4 r + k, B[k][n] at lane 4 n + k, D[r][2 q + e] at
// lane 4 r + q (element e)
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b)
{
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}
// two row tiles (d0 and d1, rows 8 apart) in one instruction, k = 4 and k = 8 (the second half at a2, a3 and b1)
__device__ __forceinline__ void dmma16(double (&d0)[2], double (&d1)[2], double a0, double a1, double b)
{
  asm("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
      : "+d"(d0[0]), "+d"(d0[1]), "+d"(d1[0]), "+d"(d1[1]) : "d"(a0), "d"(a1), "d"(b));
}
__device__ __forceinline__ void dmma16k8(double (&d0)[2], double (&d1)[2], double a0, double a1, double a2, double a3, double b0, double b1)
{
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+d"(d0[0]), "+d"(d0[1]), "+d"(d1[0]), "+d"(d1[1]) : "d"(a0), "d"(a1), "d"(a2), "d"(a3), "d"(b0), "d"(b1));
}

// row stride (doubles) of a shared-memory operand with `n4` columns (a multiple of 4) whose fragments read 4
// consecutive doubles of 8 rows: 4 or 12 mod 16 spreads a half-warp over all 16 bank pairs
__host__ __device__ constexpr int fragStride(int n4) { return n4 % 8 == 4 ? n4 : n4 + 4; }

// copies `bytes` (0, 8 or WIDTH) of a WIDTH-byte chunk and zero-fills the rest
template <int WIDTH>
__device__ __forceinline__ void cpAsync(double * dst, const double * src, int bytes)
{
  unsigned const d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  if constexpr (WIDTH == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

}  // namespace tcscf
