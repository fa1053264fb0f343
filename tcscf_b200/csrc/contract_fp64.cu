// FP64 r12 contractions and Fock-matrix reductions, on the FP64 tensor cores.
//
// The r12 contraction is written flash-style: for a tile of r1 points the kernel streams r2 in
// blocks, generates g(r1,r2) from the point coordinates (never stored), forms the density-matrix
// kernel rho(r1,r2) from the occupied-orbital factors, and accumulates  T += (g .* rho) V  in
// registers.  This reassociates the reference's stored-kernel contraction
//   Fai(r1,i) = sum_j (sum_k D(k,j) phi_k(r1)) Fji(r1,j,i),  Fji = computeF(1/r12)
// (HartreeFock.cpp:144-179, HartreeFock.hpp:136-180) into
//   Fai(r1,i) = sum_r2 g(r1,r2) w2 rho(r1,r2) phi_i(r2),  rho(r1,r2) = sum_kj D(k,j) phi_k(r1) phi_j(r2)^*
// and computes the Coulomb potential Faa(r1) (calculateIaa, HartreeFock.cpp:183-213) in the same
// pass.  With R == 0 (rho == 1) and V = weighted basis-pair products the same kernel is the FP64
// precompute form computeF / computeV.
#include "kernels.cuh"

namespace tcscf {
namespace {

constexpr int BK = 32;        // r2 points per stage
constexpr int kMaxCol = 128;  // columns per block at most

struct KArgs {
  int64_t n1, n2, r2PerSplit;
  int R, ncol, colsPerBlock, ldpsi, ldv, ldt, component, same;
  int vec16;              // V rows may be copied in 16-byte chunks
  const double * p1;
  const double * p2;
  const double * psi1;
  const double * psi2;
  const double * coul;
  const double * V;
  double * T;
  double * VH;
  int64_t tStrideSplit;   // elements between split partials of T (0 when not split)
  int64_t vhStrideSplit;
  int sym;                // r1 = r2 points and psi1 = psi2: only r2 >= the block's first row, its own rows at half weight
  OchiDev u;
};

__device__ __forceinline__ double ipow(double x, int k)
{
  double r = 1;
  for (int i = 0; i < k; ++i) r *= x;
  return r;
}

// jastrowFunctions.hpp:72-108 (Ochi::gradient) for points p (first argument) and q.
__device__ __forceinline__ void ochiGrad(OchiDev const & u, double px, double py, double pz, double qx, double qy, double qz,
                                         int same, double & gx, double & gy, double & gz)
{
  double const dx = px - qx, dy = py - qy, dz = pz - qz;
  double const r1 = sqrt(px * px + py * py + pz * pz);
  double const r2 = sqrt(qx * qx + qy * qy + qz * qz);
  double const r12 = sqrt(dx * dx + dy * dy + dz * dz);
  double const r1T = r1 / (r1 + u.a), r2T = r2 / (r2 + u.a), r12T = r12 / (r12 + u.a12);
  double const r1Scale = u.a / (r1 * r1 * (r1 + u.a));
  double const r12Scale = u.a12 / (r12 * r12 * (r12 + u.a12));
  double r1L = 0, r12L = 0;
  for (int k = 0; k < u.nterms; ++k) {
    int const i = u.S[k][0], j = u.S[k][1], kk = u.S[k][2];
    double const f = u.c[k][same] * ipow(r12T, i) * ipow(r1T, j) * ipow(r2T, kk);
    r1L += f * j * r1Scale;
    r12L += f * i * r12Scale;
  }
  gx = r12L * dx + r1L * px;
  gy = r12L * dy + r1L * py;
  gz = r12L * dz + r1L * pz;
}

// (1/r12) du/dr12 of a Jastrow factor of r12 alone (every S[k] = (i, 0, 0)) from r12^2 and y = 1/r12:
// a12 t y^2 sum_k i_k c_k (r12 t)^i_k with t = 1 / (r12 + a12); grad_1 u is this times r1 - r2
__device__ __forceinline__ double ochiR12(OchiDev const & u, double rr, double y, int same)
{
  double const r = rr * y, t = 1.0 / (r + u.a12), z = r * t;
  double s = 0;
  for (int k = 0; k < u.nterms; ++k) s = fma(u.c[k][same] * u.S[k][0], ipow(z, u.S[k][0]), s);
  return u.a12 * t * y * y * s;
}

// g(r1, r2), 0 for r1 == r2.  KIND 0 = 1/r12, 1 = TC scalar, 2 = one component of grad_1 u; 3, 4 = 1, 2 for a Jastrow factor of
// r12 alone, where grad_2 u = -grad_1 u and no other distance enters (a fifth of the FP64 operations)
template <int KIND>
__device__ __forceinline__ double r12Kernel(KArgs const & a, double x1, double y1, double z1, double x2, double y2, double z2)
{
  double const dx = x1 - x2, dy = y1 - y2, dz = z1 - z2;
  double const rr = fma(dx, dx, fma(dy, dy, dz * dz));
  if constexpr (KIND == 0) return invR12(rr);
  if constexpr (KIND == 3 || KIND == 4) {
    double const y = invR12(rr), q = y == 0.0 ? 0.0 : ochiR12(a.u, rr, y, a.same);
    if constexpr (KIND == 3) return 2.0 * (y - q * q * rr);
    return q * (a.component == 0 ? dx : (a.component == 1 ? dy : dz));
  }
  if (rr == 0.0) return 0.0;
  if (KIND == 1) {
    double ax, ay, az, bx, by, bz;
    ochiGrad(a.u, x1, y1, z1, x2, y2, z2, a.same, ax, ay, az);
    ochiGrad(a.u, x2, y2, z2, x1, y1, z1, a.same, bx, by, bz);
    return 2.0 / sqrt(rr) - (ax * ax + ay * ay + az * az) - (bx * bx + by * by + bz * bz);
  }
  double gx, gy, gz;
  ochiGrad(a.u, x1, y1, z1, x2, y2, z2, a.same, gx, gy, gz);
  return a.component == 0 ? gx : (a.component == 1 ? gy : gz);
}

// row stride of the V tile (2 mod 8: the 16-byte fragment loads below read rows 2 k + e)
__host__ __device__ constexpr int vStride(int nt) { return 8 * nt + 2; }
__host__ __device__ constexpr int contractWarps(int rt) { return rt == 1 ? 8 : 4; }

// blocks per SM the register budget is cut for (65,536 / (threads x blocks) a thread); one more block each
// below 8 tiles spilled and ran 1 to 20 % slower
__host__ __device__ constexpr int contractBlocks(int nt, int rt, int kind)
{
  return rt == 1 ? (kind == 0 ? 1 : 2) : (nt <= 3 ? 4 : (nt <= 6 ? 3 : 2));
}

// T += (g .* rho) V for 8 RT rows per warp and 8 NTL columns, everything between the shared-memory
// operands and T in registers: per 8 r2 points a warp forms rho for its rows with FP64 MMAs (psi1 psi2^T),
// whose D fragment gives each lane its row's values at points 2 q and 2 q + 1 (q = lane % 4); the lane
// multiplies them by g of the same two pairs, and the products are the A fragments of the two MMA k-steps
// that follow (step e takes the points 2 q + e, so V is read at rows 2 q + e).  X never passes through
// shared memory and no barrier separates the generation of g from the GEMM: the warps of an SM
// drift apart.  Columns are interleaved in pairs (n and n + 1 of two tiles), so one 16-byte load serves two
// MMAs.  Blocks are 4 warps (8 where RT = 1), r2 in stages of BK points through a two-stage cp.async
// pipeline.  With RT = 2 rho takes m16n8k4 MMAs and T m16n8k8 ones, with RT = 1 both take m8n8k4.  Bound by the FP64 pipe and the
// instruction issue together: an MMA takes 16 issue cycles of its scheduler per 8 x 8 x 4 product whatever its shape (32 for m16n8k4, 64 for
// m16n8k8) and nothing overlaps it, so the time is 16 x products plus the other instructions; they are kept
// few (copies without index arithmetic, the rank a template parameter, no masks in full stages, the
// half weight applied once).  Forming the next group's X beside the GEMM, MMAs of m8n8k4 and
// volatile ordering all measured the same.  Against a kernel that passed X through shared memory between
// two barriers: 59,000 points x 40 columns (rank 5, symmetric) 21.1 -> 7.2 ms; 81,200 points x 120
// columns (rank 18, symmetric) 58.6 -> 32.1 ms, 0.81 of the FP64 matmul rate counting the padded MMAs.
template <int KIND, int NTL, int RT, int KR>
__global__ void __launch_bounds__(32 * contractWarps(RT), contractBlocks(NTL, RT, KIND)) kContractFp64(KArgs a)
{
  constexpr int kWarps = contractWarps(RT), kThreads = 32 * kWarps;
  static_assert(BK == 32, "a warp copies one coordinate row of a stage");
  constexpr int BMT = 8 * RT * contractWarps(RT);   // r1 rows per block
  constexpr int VLD = vStride(NTL);
  extern __shared__ __align__(16) double sm[];
  int const R = KR == 0 ? 0 : a.R, R4 = KR >= 0 ? 4 * KR : (R + 3) / 4 * 4, pld = fragStride(R4);
  double * sP1 = sm;                                     // [BMT][pld]
  double * stage0 = sP1 + (R ? BMT * pld : 0);           // per stage: sV [BK][VLD], sC2 [4][BK], sP2 [BK][pld]
  int const stageSize = BK * VLD + 4 * BK + (R ? BK * pld : 0);

  int const tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fr = lane >> 2, fq = lane & 3;
  int64_t const r1base = int64_t(blockIdx.x) * BMT;
  int const col0 = blockIdx.z * a.colsPerBlock, ncol = min(a.ncol, col0 + a.colsPerBlock);
  // a symmetric contraction takes the r2 points from this block's own rows on (its own BMT x BMT
  // square at half weight in T); the Coulomb sums over the points before them come from kCoulombLowerFp64
  int64_t const r2split = int64_t(blockIdx.y) * a.r2PerSplit;
  int64_t const r2begin = a.sym ? max(r2split, r1base) : r2split;
  int64_t const r2end = min(a.n2, r2split + a.r2PerSplit);
  int64_t const r2half = a.sym ? r1base + BMT : 0;   // r2 below this (and >= r2begin) at half weight: whole stages, both multiples of BK
  bool const doCoul = a.coul != nullptr && blockIdx.z == 0;

  // The copies of a stage: warp w takes V and psi2 rows w, w + warps, ... (psi2: several rows at once where
  // they are short) and coordinate row w, the lanes a row's chunks; a full stage's copies differ only by
  // one pointer step from row to row, so a lane's pointers and byte counts are formed once.
  constexpr int W = 8 * NTL;
  int const cols = ncol - col0;
  // lanes of a psi2 row: at least so many that the block's rows of one step are no more than a stage's
  constexpr int kMinPsiLanes = kWarps * 32 / BK;
  static_assert(kMinPsiLanes >= 4 && kWarps * (32 / kMinPsiLanes) <= BK, "psi2 rows of a copy step within the stage");
  int const psiLanes = max(kMinPsiLanes, R4 <= 4 ? 4 : (R4 <= 8 ? 8 : (R4 <= 16 ? 16 : 32))), psiRows = 32 / psiLanes;
  int const pk = warp * psiRows + lane / psiLanes, pb = lane % psiLanes;
  int const vb0 = min(16, max(0, 8 * (cols - 2 * lane))), vb1 = min(16, max(0, 8 * (cols - 64 - 2 * lane)));
  const double * const vsrc = a.V + int64_t(warp) * a.ldv + col0 + (vb0 ? 2 * lane : 0);
  const double * const psrc = R ? a.psi2 + int64_t(pk) * a.ldpsi + (pb < R ? pb : 0) : nullptr;
  const double * const csrc = warp < 3 ? a.p2 + int64_t(warp) * a.n2 + lane : (doCoul ? a.coul + lane : a.p2 + lane);
  int64_t const vstep = int64_t(kWarps) * a.ldv, pstep = int64_t(kWarps) * psiRows * a.ldpsi;
  auto issue = [&](int64_t k0, int st) {
    double * sV = stage0 + st * stageSize;
    double * sC2 = sV + BK * VLD;
    double * sP2 = sC2 + 4 * BK;
    if (a.vec16 && R4 <= 32 && r2end - k0 >= BK) {
      const double * src = vsrc + k0 * a.ldv;
      double * dst = sV + warp * VLD + 2 * lane;
#pragma unroll
      for (int k = 0; k < BK; k += kWarps, src += vstep) {
        if (W >= 64 || 2 * lane < W) cpAsync<16>(dst + k * VLD, src, vb0);
        if (W > 64 && 64 + 2 * lane < W) cpAsync<16>(dst + k * VLD + 64, vb1 ? src + 64 : src, vb1);
      }
      if (R4 > 0 && pb < R4) {
        src = psrc + k0 * a.ldpsi;
#pragma unroll
        for (int k = 0; k < BK; k += kWarps * psiRows, src += pstep) cpAsync<8>(&sP2[(pk + k) * pld + pb], src, pb < R ? 8 : 0);
      }
      if (warp < 4) cpAsync<8>(&sC2[warp * BK + lane], csrc + k0, warp < 3 || doCoul ? 8 : 0);
      return;
    }
    int const kn = int(min(int64_t(BK), r2end - k0));
    for (int k = warp; k < BK; k += kWarps)
#pragma unroll
      for (int c = lane; c < W; c += 32) {
        bool const ok = k < kn && c < cols;
        cpAsync<8>(&sV[k * VLD + c], ok ? &a.V[(k0 + k) * a.ldv + col0 + c] : a.V, ok ? 8 : 0);
      }
    for (int k = pk; k < BK; k += kWarps * psiRows)
      for (int b = pb; b < R4; b += psiLanes) {
        bool const ok = k < kn && b < R;
        cpAsync<8>(&sP2[k * pld + b], ok ? &a.psi2[(k0 + k) * a.ldpsi + b] : a.psi2, ok ? 8 : 0);
      }
    if (warp < 4) {
      bool const ok = lane < kn && (warp < 3 || doCoul);
      cpAsync<8>(&sC2[warp * BK + lane], ok ? csrc + k0 : a.p2, ok ? 8 : 0);
    }
  };

  int64_t const nsteps = r2end > r2begin ? (r2end - r2begin + BK - 1) / BK : 0;
  if (nsteps > 0) issue(r2begin, 0);
  cpAsyncCommit();

  if constexpr (KR != 0) {
    for (int idx = tid; idx < R4 * BMT; idx += kThreads) {
      int const r = idx / R4, b = idx % R4;
      int64_t const g = r1base + r;
      sP1[r * pld + b] = b < R && g < a.n1 ? a.psi1[g * a.ldpsi + b] : 0.0;
    }
  }
  int const wrow = (tid >> 5) * 8 * RT + fr;   // this lane's row of the block in row tile 0
  double x1[RT], y1[RT], z1[RT], vh[RT];
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    int64_t const g = r1base + wrow + 8 * i;
    bool const ok = g < a.n1;
    x1[i] = ok ? a.p1[g] : 1.0e6;
    y1[i] = ok ? a.p1[a.n1 + g] : 1.0e6;
    z1[i] = ok ? a.p1[2 * a.n1 + g] : 1.0e6;
    vh[i] = 0.0;
  }
  double acc[RT][NTL][2];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  for (int64_t step = 0; step < nsteps; ++step) {
    int64_t const k0 = r2begin + step * BK;
    int const st = int(step & 1);
    __syncthreads();   // every thread is done with the stage the next issue overwrites
    if (step + 1 < nsteps) issue(k0 + BK, st ^ 1);
    cpAsyncCommit();
    cpAsyncWait<1>();
    __syncthreads();
    double const * sV = stage0 + st * stageSize;
    double const * sC2 = sV + BK * VLD;
    double const * sP2 = sC2 + 4 * BK;
    int const kn = int(min(int64_t(BK), r2end - k0));
    // the own square's stages come first: once they are in, T holds them at half weight
    if (step > 0 && k0 >= r2half && k0 - BK < r2half) {
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j) { acc[i][j][0] *= 0.5; acc[i][j][1] *= 0.5; }
    }
    // X of the 8 points from p0: x[i][e] = g rho at row tile i, point 2 q + e.  Points past kn are zeros in
    // V, psi2 and coul; 1/r12 is finite there, the transcorrelated kernels are masked
    auto generate = [&](int p0, double (&x)[RT][2]) {
#pragma unroll
      for (int i = 0; i < RT; ++i) x[i][0] = x[i][1] = R > 0 ? 0.0 : 1.0;
#pragma unroll
      for (int b = fq; b < R4 + fq; b += 4) {
        double const q = sP2[(p0 + fr) * pld + b];
        if constexpr (RT == 1) dmma(x[0], sP1[wrow * pld + b], q);
        else {
#pragma unroll
          for (int i = 0; i < RT; i += 2) dmma16(x[i], x[i + 1], sP1[(wrow + 8 * i) * pld + b], sP1[(wrow + 8 * i + 8) * pld + b], q);
        }
      }
      int const c = p0 + 2 * fq;
      double2 const px = *reinterpret_cast<double2 const *>(&sC2[c]);
      double2 const py = *reinterpret_cast<double2 const *>(&sC2[BK + c]);
      double2 const pz = *reinterpret_cast<double2 const *>(&sC2[2 * BK + c]);
      double2 const pc = *reinterpret_cast<double2 const *>(&sC2[3 * BK + c]);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        double g0 = r12Kernel<KIND>(a, x1[i], y1[i], z1[i], px.x, py.x, pz.x);
        double g1 = r12Kernel<KIND>(a, x1[i], y1[i], z1[i], px.y, py.y, pz.y);
        if constexpr (KIND != 0) {
          g0 = c < kn ? g0 : 0.0;
          g1 = c + 1 < kn ? g1 : 0.0;
        }
        vh[i] = fma(g0, pc.x, fma(g1, pc.y, vh[i]));
        x[i][0] *= g0;
        x[i][1] *= g1;
      }
    };
#pragma unroll
    for (int p0 = 0; p0 < BK; p0 += 8) {
      int const c = p0 + 2 * fq;
      double x[RT][2];
      generate(p0, x);
      // B fragments: rows 2 q (step 0) and 2 q + 1 (step 1) of this 8-point group
      double const * v = sV + c * VLD;
      auto gemm = [&](int j, double b0, double b1) {
        if constexpr (RT == 1) {
          dmma(acc[0][j], x[0][0], b0);
          dmma(acc[0][j], x[0][1], b1);
        } else {
#pragma unroll
          for (int i = 0; i < RT; i += 2) dmma16k8(acc[i][j], acc[i + 1][j], x[i][0], x[i + 1][0], x[i][1], x[i + 1][1], b0, b1);
        }
      };
#pragma unroll
      for (int j = 0; j + 1 < NTL; j += 2) {
        double2 const b0 = *reinterpret_cast<double2 const *>(&v[8 * j + 2 * fr]);
        double2 const b1 = *reinterpret_cast<double2 const *>(&v[VLD + 8 * j + 2 * fr]);
        gemm(j, b0.x, b1.x);
        gemm(j + 1, b0.y, b1.y);
      }
      if constexpr (NTL % 2) gemm(NTL - 1, v[8 * (NTL - 1) + fr], v[VLD + 8 * (NTL - 1) + fr]);
    }
  }
  double const last = nsteps > 0 && r2begin + (nsteps - 1) * BK < r2half ? 0.5 : 1.0;   // only stages of the own square

  double * T = a.T + blockIdx.y * a.tStrideSplit;
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    int64_t const g = r1base + wrow + 8 * i;
    if (g >= a.n1) continue;
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        // D column n = 2 q + e of tile j is column 8 (j - j % 2) + 2 n + j % 2 of the block (the last tile of an odd count: 8 j + n)
        int const n = 2 * fq + e;
        int const col = col0 + (NTL % 2 && j == NTL - 1 ? 8 * j + n : 8 * (j & ~1) + 2 * n + (j & 1));
        if (col < ncol) T[g * a.ldt + col] = last * acc[i][j][e];
      }
  }
  if (doCoul) {
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      double v = vh[i];
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      int64_t const g = r1base + wrow + 8 * i;
      if (fq == 0 && g < a.n1) a.VH[blockIdx.y * a.vhStrideSplit + g] = v;
    }
  }
}

// Symmetric contractions: the Coulomb row sums over the r2 points before each row's own tile (the pairs
// kContractFp64 skips): part[k][r] = sum of g(r, j) c(j) over the points j of chunk k (`chunk` points, a
// multiple of 64) with j < bm floor(r / bm), FP64 with the exact-coincidence rule and 64-term partial sums.
// One block of 64 threads per (128 rows, chunk); each thread takes rows r and r + 64 (the same bm tile, or
// consecutive 64-row tiles when bm = 64, so every condition below is uniform over the block), and the r2
// points pass through shared memory in 64-point pieces, the next piece's load in flight while the
// current one is summed.  Bound by the FP64 pipe (about 12 FP64 operations a pair); the chunks keep every
// SM busy where one block per row tile left the heaviest tiles running alone: 59,000 points (Ne) 13.8 -> 1.6 ms, 2,500 (He) 576 -> 20 us.
__global__ void __launch_bounds__(64) kCoulombLowerFp64(int64_t n, int bm, int64_t chunk, const double * __restrict__ p,
                                                       const double * __restrict__ coul, double * __restrict__ part)
{
  __shared__ double4 sq[2][64];   // x, y, z, c
  int const t = threadIdx.x;
  int64_t const r0 = int64_t(blockIdx.x) * 128 + t, r1 = r0 + 64;
  int64_t const end0 = (int64_t(blockIdx.x) * 128 / bm) * bm;   // the points before row r0's tile (a multiple of 64)
  int64_t const end1 = ((int64_t(blockIdx.x) * 128 + 64) / bm) * bm;
  // when row r1's tile starts past n, every r1 row is past n (not written): only row r0's points are read
  int64_t const begin = int64_t(blockIdx.y) * chunk, end = min(begin + chunk, end1 <= n ? end1 : end0);
  if (begin >= end) return;   // kCoulombLowerFp64Sum does not read this block's rows of part
  int64_t const a0 = r0 < n ? r0 : n - 1, a1 = r1 < n ? r1 : n - 1;   // rows past n repeat the last one (not written)
  double const x0 = p[a0], y0 = p[n + a0], z0 = p[2 * n + a0];
  double const x1 = p[a1], y1 = p[n + a1], z1 = p[2 * n + a1];
  auto load = [&](int64_t j0) { int64_t const j = j0 + t; return make_double4(p[j], p[n + j], p[2 * n + j], coul[j]); };
  sq[0][t] = load(begin);
  __syncthreads();
  double vh0 = 0.0, vh1 = 0.0;
  int buf = 0;
  for (int64_t j0 = begin; j0 < end; j0 += 64, buf ^= 1) {
    bool const more = j0 + 64 < end;
    double4 const nxt = more ? load(j0 + 64) : make_double4(0, 0, 0, 0);
    bool const row0 = j0 + 64 <= end0;
    double part0 = 0.0, part1 = 0.0;
#pragma unroll 4
    for (int e = 0; e < 64; ++e) {
      double4 const q = sq[buf][e];
      double dx = x1 - q.x, dy = y1 - q.y, dz = z1 - q.z;
      part1 = fma(invR12(fma(dx, dx, fma(dy, dy, dz * dz))), q.w, part1);
      if (row0) {
        dx = x0 - q.x; dy = y0 - q.y; dz = z0 - q.z;
        part0 = fma(invR12(fma(dx, dx, fma(dy, dy, dz * dz))), q.w, part0);
      }
    }
    vh0 += part0;
    vh1 += part1;
    if (more) sq[buf ^ 1][t] = nxt;   // the piece before's buffer: every thread finished it before the last barrier
    __syncthreads();
  }
  double * out = part + int64_t(blockIdx.y) * n;
  if (r0 < n && begin < end0) out[r0] = vh0;
  if (r1 < n && begin < end1) out[r1] = vh1;
}

// VH[r] += the row's chunk partials, in chunk order
__global__ void kCoulombLowerFp64Sum(int64_t n, int bm, int64_t chunk, const double * __restrict__ part, double * __restrict__ VH)
{
  int64_t const r = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (r >= n) return;
  int64_t const end = r / bm * bm;
  double s = 0.0;
  for (int64_t k = 0; k * chunk < end; ++k) s += part[k * n + r];
  VH[r] += s;
}

// deterministic sum of split partials: out[i] = sum_s part[s*stride + i]
__global__ void kSumSplits(int64_t n, int nsplit, int64_t stride, const double * part, double * out, int64_t rows, int cols, int ldOut, int ldPart)
{
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    int64_t const r = i / cols;
    int const c = int(i % cols);
    double s = 0.0;
    for (int k = 0; k < nsplit; ++k) s += part[k * stride + r * ldPart + c];
    out[r * ldOut + c] = s;
  }
  (void)rows;
}

// ---- real Fock reduction:  out[k][l] = sum_r w[r] phi[r][k] (cJ phi[r][l] VH[r] - T[r][l]) ----
constexpr int RB = 16;      // rows per step

struct ReduceArgs {
  int64_t n1, tStride;        // rows; elements between the spins' T
  int nb, ldt, rch;
  const double * phi;
  const double * w;
  const double * VH;          // null: no Coulomb term
  const double * T;
  double cJ[2];               // per spin
};

// One block: `rch` rows (a multiple of RB) into a W x W tile of one spin's sum, W = 8 WT Q: Q x Q warps of (8 WT)^2 on
// the FP64 tensor cores, whose fragments are 8 consecutive doubles of 4 rows (stride 4 mod 16:
// conflict-free).  Rows pass through two shared-memory stages of RB, the next stage's values loaded into registers
// while the current one is multiplied.  Q = 4 up to 128 columns reads phi and T once (Q = 2 would, above
// 64 columns, read them once per 64-wide tile).  Bound by the FP64 MMAs.  The CUDA-core form (8 x 8 outputs a
// thread, no prefetch) took, per call, 1.38 -> 1.09 ms for Kr (406,000
// points, 120 columns) and 61 -> 36 us for Ne (59,000, 40), and symmetric builds called it twice.
template <int WT, int Q>
__global__ void __launch_bounds__(32 * Q * Q) kReduceReal(ReduceArgs a, double * part)
{
  constexpr int NTH = 32 * Q * Q, W = 8 * WT * Q, LD = W % 16 == 8 ? W + 12 : W + 4, VPT = RB * W / NTH;
  static_assert(LD % 16 == 4 && RB * W % NTH == 0, "fragment stride; values per thread");
  extern __shared__ __align__(16) double sm[];
  auto sA = reinterpret_cast<double(*)[RB][LD]>(sm);   // [2][RB][LD]
  auto sY = sA + 2;
  int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fq = lane & 3;
  int const tilesW = (a.nb + W - 1) / W, spin = blockIdx.z;
  int const kg = blockIdx.y / tilesW * W, lg = blockIdx.y % tilesW * W;
  int const wk = warp / Q * 8 * WT, wl = warp % Q * 8 * WT;
  double const * T = a.T + spin * a.tStride;
  double const cJ = a.cJ[spin];
  int64_t const rbeg = int64_t(blockIdx.x) * a.rch, rend = min(a.n1, rbeg + a.rch);
  double acc[WT][WT][2];
#pragma unroll
  for (int i = 0; i < WT; ++i)
#pragma unroll
    for (int j = 0; j < WT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  double av[VPT], yv[VPT];
  auto load = [&](int64_t r0) {
#pragma unroll
    for (int q = 0; q < VPT; ++q) {
      int const idx = tid + q * NTH, c = idx % W, k = kg + c, l = lg + c;
      int64_t const r = r0 + idx / W;
      bool const in = r < rend;
      double const pk = in && k < a.nb ? a.phi[r * a.nb + k] : 0.0;
      double const pl = kg == lg ? pk : (in && l < a.nb ? a.phi[r * a.nb + l] : 0.0);
      double const t = in && l < a.nb ? T[r * a.ldt + l] : 0.0;
      av[q] = in ? a.w[r] * pk : 0.0;
      yv[q] = (in && a.VH ? cJ * pl * a.VH[r] : 0.0) - t;
    }
  };
  auto store = [&](int st) {
#pragma unroll
    for (int q = 0; q < VPT; ++q) {
      int const idx = tid + q * NTH;
      sA[st][idx / W][idx % W] = av[q];
      sY[st][idx / W][idx % W] = yv[q];
    }
  };
  if (rbeg < rend) {
    load(rbeg);
    store(0);
  }
  __syncthreads();
  int st = 0;
  for (int64_t r0 = rbeg; r0 < rend; r0 += RB, st ^= 1) {
    bool const more = r0 + RB < rend;
    if (more) load(r0 + RB);
#pragma unroll
    for (int rr = 0; rr < RB; rr += 4) {
      double af[WT], bf[WT];
#pragma unroll
      for (int i = 0; i < WT; ++i) { af[i] = sA[st][rr + fq][wk + 8 * i + fr]; bf[i] = sY[st][rr + fq][wl + 8 * i + fr]; }
#pragma unroll
      for (int i = 0; i < WT; ++i)
#pragma unroll
        for (int j = 0; j < WT; ++j) dmma(acc[i][j], af[i], bf[j]);
    }
    if (more) store(st ^ 1);   // the stage before's buffer: every warp finished it before the last barrier
    __syncthreads();
  }
  double * out = part + (int64_t(spin) * gridDim.x + blockIdx.x) * a.nb * a.nb;
#pragma unroll
  for (int i = 0; i < WT; ++i)
#pragma unroll
    for (int j = 0; j < WT; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        int const k = kg + wk + 8 * i + fr, l = lg + wl + 8 * j + 2 * fq + e;
        if (k < a.nb && l < a.nb) out[k * a.nb + l] = acc[i][j][e];
      }
}

// out[s][e] = the sum over the chunks k of part[s][k][e], e < n: 32 elements per block, 8 warps taking every eighth chunk each
// (their sums added in warp order), so that a few hundred chunks of a small matrix are not one thread's chain
__global__ void __launch_bounds__(256) kReduceSum(int n, int nchunk, const double * part, double * out)
{
  __shared__ double red[8][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  part += int64_t(blockIdx.y) * nchunk * n;
  double s = 0.0;
  if (e < n)
#pragma unroll 4
    for (int k = warp; k < nchunk; k += 8) s += part[int64_t(k) * n + e];
  red[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && e < n) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += red[k][lane];
    out[int64_t(blockIdx.y) * n + e] = s;
  }
}

template <int KIND, int NTL, int RT, int KR>
int launchOne(tcscf_ctx * ctx, KArgs const & a, dim3 grid, size_t smem)
{
  TCSCF_CUDA(ctx, cudaFuncSetAttribute(kContractFp64<KIND, NTL, RT, KR>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  TCSCF_CUDA(ctx, cudaFuncSetAttribute(kContractFp64<KIND, NTL, RT, KR>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  kContractFp64<KIND, NTL, RT, KR><<<grid, 32 * contractWarps(RT), smem, ctx->stream>>>(a);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

// the rank in steps of 4 as a template parameter where small (its loops and strides are then constants): 0 (the
// precompute form), 1, 2, 3, 5, or -1 for any other; contractSteps rounds 4 up to 5.  Against -1 for all, 16,384 x 16,000 points x
// 40 columns: rank 1 1.53 -> 1.10 ms, rank 9 1.23, rank 18 1.40; a 4 of its own would take ranks 13 to 16 from 1.39 to 1.31
// (each value is 12 more kernels to compile, so the set stops where it does)
constexpr int kAnySteps = -1;
int contractSteps(int rt, int R)
{
  int const k = (R + 3) / 4;
  return rt == 1 || k > 5 ? kAnySteps : (k == 4 ? 5 : k);
}

template <int NTL>
int launchDirect(tcscf_ctx * ctx, int kr, KArgs const & a, dim3 grid, size_t smem)
{
  switch (kr) {
    case 0: return launchOne<0, NTL, 2, 0>(ctx, a, grid, smem);
    case 1: return launchOne<0, NTL, 2, 1>(ctx, a, grid, smem);
    case 2: return launchOne<0, NTL, 2, 2>(ctx, a, grid, smem);
    case 3: return launchOne<0, NTL, 2, 3>(ctx, a, grid, smem);
    case 5: return launchOne<0, NTL, 2, 5>(ctx, a, grid, smem);
    default: return launchOne<0, NTL, 2, kAnySteps>(ctx, a, grid, smem);
  }
}

// the 8-column tiles of a block (contractTiles' result) and its row tiles per warp, as template parameters
template <int KIND>
int launchKind(tcscf_ctx * ctx, int nt, int rt, int kr, KArgs const & a, dim3 grid, size_t smem)
{
  if constexpr (KIND == 0) {
    if (rt == 1) {
      if (nt == 8) return launchOne<0, 8, 1, kAnySteps>(ctx, a, grid, smem);
      return launchOne<0, 16, 1, kAnySteps>(ctx, a, grid, smem);
    }
    switch (nt) {
      case 1: return launchDirect<1>(ctx, kr, a, grid, smem);
      case 2: return launchDirect<2>(ctx, kr, a, grid, smem);
      case 3: return launchDirect<3>(ctx, kr, a, grid, smem);
      case 4: return launchDirect<4>(ctx, kr, a, grid, smem);
      case 5: return launchDirect<5>(ctx, kr, a, grid, smem);
      case 6: return launchDirect<6>(ctx, kr, a, grid, smem);
      case 8: return launchDirect<8>(ctx, kr, a, grid, smem);
      case 10: return launchDirect<10>(ctx, kr, a, grid, smem);
      case 12: return launchDirect<12>(ctx, kr, a, grid, smem);
      case 13: return launchDirect<13>(ctx, kr, a, grid, smem);
      case 15: return launchDirect<15>(ctx, kr, a, grid, smem);
      default: return launchDirect<16>(ctx, kr, a, grid, smem);
    }
  } else {
    constexpr int RT = KIND >= 3 ? 2 : 1;
    switch (nt) {
      case 4: return launchOne<KIND, 4, RT, 0>(ctx, a, grid, smem);
      case 8: return launchOne<KIND, 8, RT, 0>(ctx, a, grid, smem);
      case 13: return launchOne<KIND, 13, RT, 0>(ctx, a, grid, smem);
      default: return launchOne<KIND, 16, RT, 0>(ctx, a, grid, smem);
    }
  }
}

// The smallest instantiated tile count that holds nt tiles.  Direct builds pay for padded tiles with MMAs: every count up to 6, then
// sets with at most one padded tile (16,384 x 16,000 points, rank 5, with / without a kernel of its own: 7 tiles 1.49 / 1.63 ms, 9 1.75 /
// 1.87, 11 2.05 / 2.13, 14 2.38 / 2.60; counts of 4, 8 and 16 alone 0.95 for 1 tile's 0.55, 2.57 for 9).  The transcorrelated kernels'
// time is g first: four counts, 13 being the three groups of the 300 pair products of 24 functions (8,192 x 8,000 points: 3.10 ms, with 16 tiles 3.36);
// the padding of 9 tiles to 13 costs them 13 to 17 %, of 6 to 8 2 to 30 %.  More of either is compile time: all 16 counts double it.
// Eight warps of one row tile: factors too wide for the shared memory of two, which only bases above 32 columns (8 or 16 tiles) have
int contractTiles(int kind, int rt, int nt)
{
  static int const direct[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 13, 15, 16}, wideRank[] = {8, 16}, tc[] = {4, 8, 13, 16};
  auto pick = [&](auto const & v) { for (int t : v) if (t >= nt) return t; return 16; };
  return kind != 0 ? pick(tc) : (rt == 1 ? pick(wideRank) : pick(direct));
}

size_t contractSmem(int nt, int rt, int R)
{
  int const kr = contractSteps(rt, R), bm = 8 * rt * contractWarps(rt), p = R > 0 ? fragStride(kr > 0 ? 4 * kr : (R + 3) / 4 * 4) : 0;
  return sizeof(double) * (size_t(bm) * p + 2 * (size_t(BK) * vStride(nt) + 4 * BK + size_t(BK) * p));
}

}  // namespace

int contractFp64(tcscf_ctx * ctx, Contraction const & c)
{
  TCSCF_CHECK(ctx, c.R >= 0 && c.R <= 128, TCSCF_ERR_UNSUPPORTED, "contraction rank must be <= 128");
  TCSCF_CHECK(ctx, c.ncol > 0 && c.n1 > 0 && c.n2 > 0, TCSCF_ERR_INVALID_ARGUMENT, "empty contraction");
  bool r12Only = c.jastrow != nullptr;
  for (int k = 0; r12Only && k < c.jastrow->nterms; ++k) r12Only = c.jastrow->S[k][1] == 0 && c.jastrow->S[k][2] == 0 && c.jastrow->S[k][0] >= 0;
  int const kind = c.kernel == TCSCF_K_INV_R12 ? 0 : (c.kernel <= TCSCF_K_TC_SCALAR_OPPO ? 1 : 2) + (r12Only ? 2 : 0);
  TCSCF_CHECK(ctx, kind == 0 || c.R == 0, TCSCF_ERR_UNSUPPORTED, "internal: the transcorrelated kernels come in the precompute form");
  // columns in equal groups of at most 128 (g is generated once per group)
  int const cgroups = (c.ncol + kMaxCol - 1) / kMaxCol;
  int const colsPerBlock = ((c.ncol + cgroups - 1) / cgroups + 7) / 8 * 8;
  // two row tiles per warp (with four, 59,000 points x 40 columns took 9.8 ms against 8.5: half the warps, and
  // the accumulators spilled); ranks whose factor rows would leave room for one block of 4 warps per
  // SM take 8 warps of one row tile, and so do the general transcorrelated kernels, whose long chains of roots and
  // quotients want 16 warps per SM
  int rt = kind == 1 || kind == 2 ? 1 : 2;
  if (kind == 0 && contractSmem(contractTiles(kind, rt, colsPerBlock / 8), rt, c.R) > 112 * 1024) rt = 1;
  int const nt = contractTiles(kind, rt, colsPerBlock / 8);
  int const bm = 8 * rt * contractWarps(rt);
  int64_t const tiles = (c.n1 + bm - 1) / bm;
  int dev = 0;
  cudaGetDevice(&dev);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // split r2 so that there are several waves of blocks (2 to 3 per SM; a symmetric contraction's first
  // tiles take the whole range and its last ones almost nothing): partials are summed deterministically, and
  // kept below 512 MiB
  int64_t const want = int64_t(sms) * (c.sym ? 24 : 12);
  int64_t nsplit = (want + tiles * cgroups - 1) / (tiles * cgroups);
  nsplit = std::min<int64_t>(nsplit, (int64_t(512) << 20) / (c.n1 * c.ldt * int64_t(sizeof(double))));
  nsplit = std::max<int64_t>(1, std::min<int64_t>(nsplit, (c.n2 + 4 * BK - 1) / (4 * BK)));
  nsplit = std::min<int64_t>(nsplit, 65535);
  int64_t perSplit = (c.n2 + nsplit - 1) / nsplit;
  perSplit = ((perSplit + BK - 1) / BK) * BK;
  nsplit = (c.n2 + perSplit - 1) / perSplit;

  KArgs a{};
  a.n1 = c.n1; a.n2 = c.n2; a.r2PerSplit = perSplit;
  a.R = c.R; a.ncol = c.ncol; a.colsPerBlock = colsPerBlock; a.ldpsi = c.ldpsi; a.ldv = c.ldv; a.ldt = c.ldt;
  a.component = c.component; a.same = (c.kernel == TCSCF_K_TC_SCALAR_SAME || c.kernel == TCSCF_K_GRAD_U_SAME) ? 1 : 0;
  a.p1 = c.p1; a.p2 = c.p2; a.psi1 = c.psi1; a.psi2 = c.psi2; a.coul = c.coul; a.V = c.V;
  if (c.jastrow) {
    a.u.a = c.jastrow->a; a.u.a12 = c.jastrow->a12; a.u.nterms = c.jastrow->nterms;
    for (int k = 0; k < 8; ++k) {
      for (int d = 0; d < 3; ++d) a.u.S[k][d] = c.jastrow->S[k][d];
      a.u.c[k][0] = c.jastrow->c[k][0]; a.u.c[k][1] = c.jastrow->c[k][1];
    }
  }
  double * Tpart = c.T;
  double * VHpart = c.VH;
  if (nsplit > 1) {
    void * p = nullptr;
    size_t const tb = size_t(nsplit) * c.n1 * c.ldt * sizeof(double);
    size_t const vb = c.coul ? size_t(nsplit) * c.n1 * sizeof(double) : 0;
    TCSCF_TRY(scratch(ctx, "contract_split", tb + vb, &p));
    Tpart = static_cast<double *>(p);
    VHpart = c.coul ? Tpart + size_t(nsplit) * c.n1 * c.ldt : nullptr;
    a.tStrideSplit = c.n1 * c.ldt;
    a.vhStrideSplit = c.n1;
  }
  a.T = Tpart;
  a.VH = VHpart;
  TCSCF_CHECK(ctx, !c.sym || (c.p1 == c.p2 && c.n1 == c.n2 && c.psi1 == c.psi2 && c.R > 0 && (c.VH != nullptr) == (c.coul != nullptr)),
              TCSCF_ERR_INVALID_ARGUMENT, "internal: a symmetric contraction needs r1 = r2 and psi1 = psi2");
  a.sym = c.sym ? 1 : 0;
  // 16-byte copies of V: every chunk starts at an even column of a 16-byte aligned row
  a.vec16 = c.ldv % 2 == 0 && reinterpret_cast<uintptr_t>(c.V) % 16 == 0;
  size_t const smem = contractSmem(nt, rt, c.R);
  TCSCF_CHECK(ctx, smem <= 227 * 1024, TCSCF_ERR_UNSUPPORTED, "internal: contraction tile beyond the shared memory");
  // the contraction kernel alone is bracketed by the context's timing events (tcscf_last_timing)
  if (!ctx->capturing) cudaEventRecord(ctx->evStart(), ctx->stream);
  dim3 const grid{unsigned(tiles), unsigned(nsplit), unsigned(cgroups)};
  switch (kind) {
    case 0: TCSCF_TRY(launchKind<0>(ctx, nt, rt, contractSteps(rt, c.R), a, grid, smem)); break;
    case 1: TCSCF_TRY(launchKind<1>(ctx, nt, rt, 0, a, grid, smem)); break;
    case 2: TCSCF_TRY(launchKind<2>(ctx, nt, rt, 0, a, grid, smem)); break;
    case 3: TCSCF_TRY(launchKind<3>(ctx, nt, rt, 0, a, grid, smem)); break;
    default: TCSCF_TRY(launchKind<4>(ctx, nt, rt, 0, a, grid, smem)); break;
  }
  if (!ctx->capturing) cudaEventRecord(ctx->evStop(), ctx->stream);
  if (nsplit > 1) {
    int64_t const n = c.n1 * c.ncol;
    kSumSplits<<<gridBlocks(n, 256), 256, 0, ctx->stream>>>(n, int(nsplit), c.n1 * c.ldt, Tpart, c.T, c.n1, c.ncol, c.ldt, c.ldt);
    TCSCF_LAUNCH(ctx);
    if (c.coul) {
      kSumSplits<<<gridBlocks(c.n1, 256), 256, 0, ctx->stream>>>(c.n1, int(nsplit), c.n1, VHpart, c.VH, c.n1, 1, 1, 1);
      TCSCF_LAUNCH(ctx);
    }
  }
  if (c.sym && c.coul && tiles > 1) {
    // about 16 blocks of row tiles and chunks per resident block slot (half of them lie above the diagonal
    // and return at once), at least 64 points a chunk
    int64_t const rows = (c.n1 + 127) / 128;
    int64_t const want = std::max<int64_t>(8, (int64_t(sms) * 256 + rows - 1) / rows);
    int64_t const chunk = std::max<int64_t>(64, (c.n1 + want - 1) / want / 64 * 64);
    int64_t const chunks = (c.n1 + chunk - 1) / chunk;
    void * p = nullptr;
    TCSCF_TRY(scratch(ctx, "coulomb_lower", size_t(chunks) * c.n1 * sizeof(double), &p));
    double * part = static_cast<double *>(p);
    kCoulombLowerFp64<<<dim3(unsigned(rows), unsigned(chunks)), 64, 0, ctx->stream>>>(c.n1, bm, chunk, c.p1, c.coul, part);
    TCSCF_LAUNCH(ctx);
    kCoulombLowerFp64Sum<<<unsigned((c.n1 + 255) / 256), 256, 0, ctx->stream>>>(c.n1, bm, chunk, part, c.VH);
    TCSCF_LAUNCH(ctx);
  }
  return TCSCF_OK;
}

int sumSplitsLaunch(tcscf_ctx * ctx, int64_t n, int nsplit, int64_t stride, const double * part, double * out, int64_t rows, int cols,
                    int ldOut, int ldPart)
{
  kSumSplits<<<gridBlocks(n, 256), 256, 0, ctx->stream>>>(n, nsplit, stride, part, out, rows, cols, ldOut, ldPart);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

int reduceFockReal(tcscf_ctx * ctx, int64_t n1, int nb, int nspin, const double * phi, const double * w1, const double * VH,
                   const double * cJ, const double * T, int64_t tStride, int ldt, double * out)
{
  // tiles 16, 32, 48 or 64 wide with 4 warps up to 64 columns, 96 or 128 wide with 16 warps above: the least padding
  int const Q = nb <= 64 ? 2 : 4;
  int const wt = Q == 2 ? (nb + 15) / 16 : (nb <= 96 ? 3 : 4);
  int const W = 8 * wt * Q, g = (nb + W - 1) / W;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  // row chunks for four small or two large blocks per SM (16 to 1024 rows a chunk)
  int64_t const blocks = std::max<int64_t>(1, (Q == 2 ? 4 : 2) * int64_t(sms) / (int64_t(g) * g * nspin));
  int64_t const rows = (n1 + blocks - 1) / blocks;
  int const rch = int(std::min<int64_t>(1024, std::max<int64_t>(RB, (rows + RB - 1) / RB * RB)));
  int64_t const chunks = (n1 + rch - 1) / rch;
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "reduce_real", size_t(nspin) * chunks * nb * nb * sizeof(double), &p));
  double * part = static_cast<double *>(p);
  ReduceArgs a{n1, tStride, nb, ldt, rch, phi, w1, VH, T, {cJ[0], nspin > 1 ? cJ[1] : 0.0}};
  dim3 const grid{unsigned(chunks), unsigned(g * g), unsigned(nspin)};
  auto launch = [&](auto kernel) {
    size_t const smem = sizeof(double) * 4 * RB * (W % 16 == 8 ? W + 12 : W + 4);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    kernel<<<grid, 32 * Q * Q, smem, ctx->stream>>>(a, part);
  };
  if (Q == 2) {
    if (wt == 1) launch(kReduceReal<1, 2>);
    else if (wt == 2) launch(kReduceReal<2, 2>);
    else if (wt == 3) launch(kReduceReal<3, 2>);
    else launch(kReduceReal<4, 2>);
  } else if (wt == 3) launch(kReduceReal<3, 4>);
  else launch(kReduceReal<4, 4>);
  TCSCF_LAUNCH(ctx);
  int const n = nb * nb;
  kReduceSum<<<dim3(unsigned((n + 31) / 32), unsigned(nspin)), 256, 0, ctx->stream>>>(n, int(chunks), part, out);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

}  // namespace tcscf
