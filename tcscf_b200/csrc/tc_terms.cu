// Transcorrelated (TC) per-iteration Fock build and the TC SCF driver (FP64).
//
// TCHartreeFock (HartreeFock.cpp:102-609 per-point terms, :1105-1261 iteration, :1150-1224 assembly)
// builds, from the stored scalar tensors Fji (same / opposite spin TC kernels, computeF) and the
// vector tensors Vji (grad u, computeV) on the r1 grid:
//   G2 = two-body scalar + (vector - vector^dagger) terms,  G3 = three-body term,
//   F = h + G2 - G3,  E = sum D(i,j) (h + G2/2 - G3/3)(j,i)                        (HartreeFock.cpp:83-92)
// Each per-point intermediate of the reference (scaled gradients, Vai, Vja, Vjb, Vab norms, V-tilde,
// V-tilde_i, sum_b V_bi . V-tilde_b, occupied density, sum_b conj(V-tilde_b) occ_b) is one kernel
// over (spin, r1[, i]) here; the (j, i) matrix elements are block reductions over r1.  The SCF
// step solves the non-Hermitian pencil F C = S C e on the GPU: S = L L^H (cuSOLVER potrf),
// L^-1 F L^-H (cuBLAS trsm), the general eigen-solve cusolverDnXgeev, C = L^-H Y; then, as the
// reference does (:1298-1353), eigenvalues are sorted by real part and the occupied vectors are
// orthogonalised with the S-metric modified Gram-Schmidt of orthogonalization.hpp:136-154, whose
// vectors after the first are normalised with the Euclidean norm (:152).
#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include <cublas_v2.h>

#include "kernels.cuh"
#include "tc_device.cuh"

namespace tcscf {
namespace {

struct Z3 {
  double2 x, y, z;
};

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 zscale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
__device__ __forceinline__ Z3 z3load(const double2 * p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ void z3store(double2 * p, Z3 const & a) { p[0] = a.x; p[1] = a.y; p[2] = a.z; }
__device__ __forceinline__ Z3 z3zero() { return {make_double2(0, 0), make_double2(0, 0), make_double2(0, 0)}; }
__device__ __forceinline__ void z3axpy(Z3 & a, double2 s, Z3 const & b)
{
  a.x = zadd(a.x, zmul(s, b.x));
  a.y = zadd(a.y, zmul(s, b.y));
  a.z = zadd(a.z, zmul(s, b.z));
}
__device__ __forceinline__ double2 z3dot(Z3 const & a, Z3 const & b) { return zadd(zadd(zmul(a.x, b.x), zmul(a.y, b.y)), zmul(a.z, b.z)); }
__device__ __forceinline__ Z3 z3conj(Z3 const & a) { return {zconj(a.x), zconj(a.y), zconj(a.z)}; }
__device__ __forceinline__ double z3norm(Z3 const & a)
{
  return a.x.x * a.x.x + a.x.y * a.x.y + a.y.x * a.y.x + a.y.y * a.y.y + a.z.x * a.z.x + a.z.y * a.z.y;
}

struct R3 {
  double x, y, z;
};
__device__ __forceinline__ double2 zrfma(double a, double2 b, double2 c) { return make_double2(fma(a, b.x, c.x), fma(a, b.y, c.y)); }
__device__ __forceinline__ void z3axpy(Z3 & a, double2 s, R3 const & b)
{
  a.x = zrfma(b.x, s, a.x);
  a.y = zrfma(b.y, s, a.y);
  a.z = zrfma(b.z, s, a.z);
}
__device__ __forceinline__ double2 z3dot(R3 const & a, Z3 const & b) { return zrfma(a.x, b.x, zrfma(a.y, b.y, zscale(a.z, b.z))); }

// Device view of one TC build in the real-harmonic basis: inputs (the kept tensors' planes as they are) and the
// per-point intermediates ([2] = spin).
struct TcView {
  int64_t n1;
  int nb, nelMax, ld, ps;                // ld, ps: tensorStride(nb), tensorPlane(nb)
  int nel[2];
  const double * Fs;                     // [n1][ps]
  const double * Fo;
  const double * Vs;                     // [n1][3][ps]
  const double * Vo;
  const double * vals;                   // [n1][nb]
  const double2 * grads;                 // [n1][nb][3]
  const double * w;                      // [n1]
  const double2 * D;                     // [2][nb][nb], D_s(i,j) at [s][i][j]
  const double2 * C0;                    // occupied orbitals of spin 0: (i, b) at [b*nb + i]
  const double2 * C1;
  double2 * Faa;                         // [2][n1]
  double2 * Fai;                         // [2][n1][nb]
  double2 * VT;                          // [2][n1][3]   V-tilde (= VaaSPO)
  double2 * SG;                          // [2][n1][3]   scaled gradients
  double * occD;                         // [2][n1]
  double2 * Vai;                         // [2][n1][nb]
  double2 * Vja;                         // [2][n1][nb][3]
  double2 * VTs;                         // [2][n1][nb][3] V-tilde_i
  double2 * Vjbs;                        // [2][n1][nb][nelMax][3]
  double2 * Vjbo;
  double * sumNs;                        // [2][n1]
  double * sumNo;
  double2 * SVD;                         // [2][n1][nb]  sum_b V_bi . V-tilde_b
  double2 * SCV;                         // [2][n1][3]   sum_b conj(V-tilde_b) occ_b
};

__device__ __forceinline__ double fget(TcView const & t, const double * F, int64_t r, int j, int i) { return F[r * t.ps + j * t.ld + i]; }
__device__ __forceinline__ R3 vget(TcView const & t, const double * V, int64_t r, int j, int i)
{
  const double * p = V + 3 * r * t.ps + j * t.ld + i;
  return {p[0], p[t.ps], p[2 * t.ps]};
}
__device__ __forceinline__ double2 dget(TcView const & t, int s, int i, int j) { return t.D[(int64_t(s) * t.nb + i) * t.nb + j]; }
__device__ __forceinline__ double2 cget(TcView const & t, int s, int i, int b) { return (s == 0 ? t.C0 : t.C1)[int64_t(b) * t.nb + i]; }
__device__ __forceinline__ Z3 gget(TcView const & t, int64_t r, int k) { return z3load(t.grads + (r * t.nb + k) * 3); }

#define TC_GRID_LOOP(total) for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < (total); idx += int64_t(gridDim.x) * blockDim.x)

// per r1, both spins: Faa (calculateIaa on both Fji, :1119-1124), V-tilde (calculateIaa on Vji :1125-1126
// and calculateVTilde :397-434 are the same sum), scaled gradients (:102-140), occupied density (:530-567).  A warp per
// point, the lanes over the elements (i, j) of its planes: F(j,i) D(i,j) = F(i,j) D(i,j) element by element, the planes being
// symmetric.  A thread per (spin, point), each walking the eight planes of its own: 65,536 points 13.6 -> 1.1 ms (33 functions), 59 -> 3.8 (64)
__global__ void __launch_bounds__(128) kTcPoint(TcView t)
{
  int const nb = t.nb, lane = threadIdx.x & 31;
  for (int64_t r = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; r < t.n1; r += int64_t(gridDim.x) * blockDim.x >> 5) {
    double2 faa[2], occ[2];
    Z3 vt[2], sg[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      faa[s] = occ[s] = make_double2(0, 0);
      vt[s] = sg[s] = z3zero();
    }
    for (int e = lane; e < nb * t.ld; e += 32) {
      int const i = e / t.ld, j = e - i * t.ld;
      if (j >= nb) continue;
      double2 const d[2] = {dget(t, 0, i, j), dget(t, 1, i, j)};
      double const fs = fget(t, t.Fs, r, i, j), fo = fget(t, t.Fo, r, i, j), vj = t.vals[r * nb + j], vi = t.vals[r * nb + i];
      R3 const vs = vget(t, t.Vs, r, i, j), vo = vget(t, t.Vo, r, i, j);
      Z3 const g = gget(t, r, i);
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        faa[s] = zrfma(fs, d[s], zrfma(fo, d[1 - s], faa[s]));
        z3axpy(vt[s], d[s], vs);
        z3axpy(vt[s], d[1 - s], vo);
        z3axpy(sg[s], zscale(vj, d[s]), g);
        occ[s] = zrfma(vj * vi, d[s], occ[s]);
      }
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      double * const v[15] = {&faa[s].x, &faa[s].y, &vt[s].x.x, &vt[s].x.y, &vt[s].y.x, &vt[s].y.y, &vt[s].z.x, &vt[s].z.y,
                              &sg[s].x.x, &sg[s].x.y, &sg[s].y.x, &sg[s].y.y, &sg[s].z.x, &sg[s].z.y, &occ[s].x};
#pragma unroll
      for (int q = 0; q < 15; ++q)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) *v[q] += __shfl_xor_sync(0xffffffffu, *v[q], o);
      if (lane == 0) {
        int64_t const idx = s * t.n1 + r;
        t.Faa[idx] = faa[s];
        z3store(t.VT + idx * 3, vt[s]);
        z3store(t.SG + idx * 3, sg[s]);
        t.occD[idx] = occ[s].x;
      }
    }
  }
}

// per (spin, r1, i): Fai (calculateFai, :1127), Vai (:217-252), Vja (:256-291, row j = i here) and
// V-tilde_i (:438-480)
__global__ void kTcPointI(TcView t)
{
  int const nb = t.nb;
  TC_GRID_LOOP(2 * t.n1 * nb)
  {
    int const i = int(idx % nb);
    int64_t const sr = idx / nb;
    int const s = int(sr / t.n1);
    int64_t const r = sr % t.n1;
    double2 fai = make_double2(0, 0), vai = make_double2(0, 0);
    Z3 vts = z3zero(), vja = z3zero();
    for (int j = 0; j < nb; ++j) {
      double2 kv = make_double2(0, 0), kc = make_double2(0, 0);
      Z3 kg = z3zero();
      for (int k = 0; k < nb; ++k) {
        kv = zrfma(t.vals[r * nb + k], dget(t, s, k, j), kv);
        z3axpy(kg, dget(t, s, k, j), gget(t, r, k));
        kc = zrfma(t.vals[r * nb + k], dget(t, s, j, k), kc);
      }
      R3 const vji = vget(t, t.Vs, r, j, i);
      fai = zrfma(fget(t, t.Fs, r, j, i), kv, fai);
      vai = zadd(vai, z3dot(vji, kg));
      z3axpy(vts, kv, vji);                              // sum_k (sum_l D(l,k) v_l) V(k,i), k := j
      z3axpy(vja, kc, vji);                              // row i of Vja: sum_j (sum_k D(j,k) v_k) V(i,j), V symmetric
    }
    t.Fai[idx] = fai;
    t.Vai[idx] = vai;
    z3store(t.VTs + idx * 3, vts);
    z3store(t.Vja + idx * 3, vja);
  }
}

// per (spin, r1, j, b < nel): Vjb for the same- and opposite-spin tensors (calculateVjb, :295-337)
__global__ void kTcVjb(TcView t)
{
  int const nb = t.nb, nm = t.nelMax;
  TC_GRID_LOOP(2 * t.n1 * nb * nm)
  {
    int const b = int(idx % nm);
    int64_t k = idx / nm;
    int const j = int(k % nb);
    k /= nb;
    int const s = int(k / t.n1);
    int64_t const r = k % t.n1;
    Z3 rs = z3zero(), ro = z3zero();
    if (b < t.nel[s]) {
      for (int i = 0; i < nb; ++i) {
        double2 const c = cget(t, s, i, b);
        z3axpy(rs, c, vget(t, t.Vs, r, i, j));   // V(j,i), read so that the lanes' j are adjacent
        z3axpy(ro, c, vget(t, t.Vo, r, i, j));
      }
    }
    z3store(t.Vjbs + idx * 3, rs);
    z3store(t.Vjbo + idx * 3, ro);
  }
}

// per (spin, r1): sum_ab |Vab|^2 for both tensors (calculateVab, :341-393), and
// sum_b conj(V-tilde_b) occ_b (:571-609)
__global__ void kTcVab(TcView t)
{
  int const nb = t.nb, nm = t.nelMax;
  TC_GRID_LOOP(2 * t.n1)
  {
    int const s = int(idx / t.n1);
    int64_t const r = idx % t.n1;
    int const ne = t.nel[s];
    double ns = 0, no = 0;
    for (int a = 0; a < ne; ++a)
      for (int b = 0; b < ne; ++b) {
        Z3 rs = z3zero(), ro = z3zero();
        for (int j = 0; j < nb; ++j) {
          double2 const cc = zconj(cget(t, s, j, a));
          int64_t const o = ((idx * nb + j) * nm + b) * 3;
          z3axpy(rs, cc, z3load(t.Vjbs + o));
          z3axpy(ro, cc, z3load(t.Vjbo + o));
        }
        ns += z3norm(rs);
        no += z3norm(ro);
      }
    t.sumNs[idx] = ns;
    t.sumNo[idx] = no;
    Z3 cs = z3zero();
    for (int k = 0; k < nb; ++k) {
      Z3 const vk = z3conj(z3load(t.VTs + (idx * nb + k) * 3));
      for (int l = 0; l < nb; ++l) z3axpy(cs, zscale(t.vals[r * nb + l], dget(t, s, l, k)), vk);
    }
    z3store(t.SCV + idx * 3, cs);
  }
}

// per (spin, r1, i): sum_k V(k,i) . (sum_l D(l,k) V-tilde_l)   (calculateSumOverb_Vbi_dot_VTildeb, :484-526)
__global__ void kTcSvd(TcView t)
{
  int const nb = t.nb;
  TC_GRID_LOOP(2 * t.n1 * nb)
  {
    int const i = int(idx % nb);
    int64_t const sr = idx / nb;
    int const s = int(sr / t.n1);
    int64_t const r = sr % t.n1;
    double2 acc = make_double2(0, 0);
    for (int k = 0; k < nb; ++k) {
      Z3 ell = z3zero();
      for (int l = 0; l < nb; ++l) z3axpy(ell, dget(t, s, l, k), z3load(t.VTs + (sr * nb + l) * 3));
      acc = zadd(acc, z3dot(vget(t, t.Vs, r, k, i), ell));
    }
    t.SVD[idx] = acc;
  }
}

// one block per (spin, j, i): the r1 sums of the scalar, vector and three-body terms (:1150-1216);
// out[0] = scalar, out[1] = vector, out[2] = scalar3, each [2][nb][nb]
__global__ void kTcReduce(TcView t, double2 * out)
{
  int const nb = t.nb, nn = nb * nb, nm = t.nelMax;
  int const s = blockIdx.x / nn, so = 1 - s, ji = blockIdx.x % nn, j = ji / nb, i = ji % nb;
  int const ne = t.nel[s];
  double2 sc = make_double2(0, 0), ve = make_double2(0, 0), s3 = make_double2(0, 0);
  for (int64_t r = threadIdx.x; r < t.n1; r += blockDim.x) {
    int64_t const ps = int64_t(s) * t.n1 + r, po = int64_t(so) * t.n1 + r;
    double const w = t.w[r];
    double const vi = t.vals[r * nb + i], vj = t.vals[r * nb + j];
    Z3 const gi = gget(t, r, i);
    R3 const vsji = vget(t, t.Vs, r, j, i), voji = vget(t, t.Vo, r, j, i);
    // two-body scalar
    sc = zadd(sc, zscale(w * vj, zsub(zscale(vi, t.Faa[ps]), t.Fai[ps * nb + i])));
    // two-body vector
    Z3 const vt = z3load(t.VT + ps * 3), vto = z3load(t.VT + po * 3);
    double2 va = zscale(vj, zsub(z3dot(vt, gi), t.Vai[ps * nb + i]));
    va = zadd(va, z3dot(vsji, z3load(t.SG + ps * 3)));
    va = zadd(va, z3dot(voji, z3load(t.SG + po * 3)));
    va = zsub(va, z3dot(z3load(t.Vja + (ps * nb + j) * 3), gi));
    ve = zadd(ve, zscale(w, va));
    // three-body
    Z3 const vti = z3load(t.VTs + (ps * nb + i) * 3), vtj = z3load(t.VTs + (ps * nb + j) * 3);
    double2 x = make_double2((z3norm(vt) - t.sumNs[ps] - t.sumNo[po]) * vj * vi, 0.0);
    x = zadd(x, zscale(2.0 * vj, zsub(t.SVD[ps * nb + i], z3dot(vt, vti))));
    x = zadd(x, zscale(2.0 * vi, zsub(zconj(t.SVD[ps * nb + j]), z3dot(z3conj(vtj), vt))));
    double2 sbS = make_double2(0, 0), sbO = make_double2(0, 0);
    for (int b = 0; b < ne; ++b) {
      int64_t const oj = ((ps * nb + j) * nm + b) * 3, oi = ((ps * nb + i) * nm + b) * 3;
      sbS = zadd(sbS, z3dot(z3load(t.Vjbs + oj), z3conj(z3load(t.Vjbs + oi))));
      sbO = zadd(sbO, z3dot(z3load(t.Vjbo + oj), z3conj(z3load(t.Vjbo + oi))));
    }
    x = zadd(x, zscale(2.0 * t.occD[ps], zsub(z3dot(vsji, vt), sbS)));
    x = zadd(x, zscale(2.0, zsub(z3dot(vti, z3conj(vtj)), z3dot(vsji, z3load(t.SCV + ps * 3)))));
    x = zadd(x, zscale(2.0 * t.occD[po], zsub(z3dot(voji, vto), sbO)));
    x = zsub(x, zscale(2.0, z3dot(voji, z3load(t.SCV + po * 3))));
    s3 = zadd(s3, zscale(w, x));
  }
  double v[6] = {sc.x, sc.y, ve.x, ve.y, s3.x, s3.y};
#pragma unroll
  for (int q = 0; q < 6; ++q)
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  __shared__ double red[6][32];
  int const lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0)
    for (int q = 0; q < 6; ++q) red[q][wid] = v[q];
  __syncthreads();
  if (threadIdx.x == 0) {
    double a[6] = {0, 0, 0, 0, 0, 0};
    for (int k = 0; k < int(blockDim.x >> 5); ++k)
      for (int q = 0; q < 6; ++q) a[q] += red[q][k];
    for (int q = 0; q < 3; ++q) out[int64_t(q) * 2 * nn + blockIdx.x] = make_double2(a[2 * q], a[2 * q + 1]);
  }
}

// G2 = scalar/2 + vec - vec^dagger with vec = vector/2, G3 = scalar3/2; masked where h == 0 when
// respectSym (enforceOneElectronSymmetry, :758-780)
__global__ void kTcAssemble(int nb, const double2 * sums, const double * h, int respectSym, double2 * G2, double2 * G3)
{
  int const nn = nb * nb;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < 2 * nn; idx += gridDim.x * blockDim.x) {
    int const s = idx / nn, ji = idx % nn, j = ji / nb, i = ji % nb;
    double2 const scal = sums[idx], vec = sums[2 * nn + idx], vecT = sums[2 * nn + s * nn + i * nb + j], s3 = sums[4 * nn + idx];
    double2 g2 = make_double2(0.5 * scal.x + 0.5 * vec.x - 0.5 * vecT.x, 0.5 * scal.y + 0.5 * vec.y + 0.5 * vecT.y);
    double2 g3 = make_double2(0.5 * s3.x, 0.5 * s3.y);
    if (respectSym && !(fabs(h[ji]) > 0)) { g2 = make_double2(0, 0); g3 = make_double2(0, 0); }
    G2[idx] = g2;
    G3[idx] = g3;
  }
}

// column-major copy of a row-major square matrix (out(j,i) = in[j][i])
__global__ void kToColMajorZ(int nb, const double2 * in, double2 * out)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nb; idx += gridDim.x * blockDim.x) {
    int const j = idx / nb, i = idx % nb;
    out[i * nb + j] = in[idx];
  }
}
__global__ void kRealToZ(int n, const double * in, double2 * out)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) out[idx] = make_double2(in[idx], 0.0);
}

// ---- fused per-point build (nb <= kFusedMaxNb) -------------------------------------------------------
// Both forms of the build work on the tensors as they are kept: real symmetric [nb][nb] planes in the real-harmonic
// basis, where the basis values are real too and only densities, orbitals and gradients are complex
// (every term pairs one conjugated and one plain index, so the sums transform back as one matrix each,
// kSumsToReference).  The kernels above keep every per-point intermediate in HBM and read the tensors several times
// over; kTcFused reads them once.  A block walks the points p = block, block + grid, ...; one point's planes (Vs, Vo
// components, Fs, Fo) arrive in shared memory by bulk copies while the block before them is still at its
// outer products.  Everything that is a contraction runs on the FP64 tensor cores:
//   (1) V(j,i) x_i for all vectors x at once (columns: sum_k D(k,i) v_k, sum_k D(i,k) v_k, sum_k D(k,i) g_k and the
//       occupied orbitals of both spins), and Fs(j,i) x_i
//   (2) the traces of the 8 planes with both densities: [8][nb^2] x [nb^2][4]
//   (3) V(j,i) ell_i
//   (4) the terms V(j,i) W linear in the planes, accumulated over the points: [nb (nb+1)/2][8] x [8][8]
//   (5) the outer products of per-point vectors, accumulated over the points: per spin a [nb][K] x [K][nb] product
//       for the scalar (K = 1 complex term), vector (4) and three-body sums (5 + 6 nel); k rows are re and im parts, the
//       fragments of the real and the imaginary result plain 8-byte loads with the sign in A's weight.
// The (spin, j tile) warps keep (5)'s accumulators, the others (4)'s, in registers over all points.  Terms, with
// v, g the point's basis values and gradients, occ_s the occupied density:
//   scalar  w v_j (Faa v_i - Fai_i)
//   vector  w v_j (VT.g_i - Vai_i) - w Vja_j . g_i + w (Vs(j,i).SG_s + Vo(j,i).SG_o)
//   three   w v_j ((|VT|^2 - sumN_s - sumN_o) v_i + 2 SVD_i - 2 VT.VTs_i) + 2w (conj(SVD_j) - conj(VTs_j).VT) v_i
//           + 2w conj(VTs_j).VTs_i - 2w occ_s Vjbs_jb . conj(Vjbs_ib) - 2w occ_o Vjbo_jb . conj(Vjbo_ib)
//           + w Vs(j,i).(2 occ_s VT_s - 2 SCV_s) + w Vo(j,i).(2 occ_o VT_o - 2 SCV_o)
// The per-block sums go to part[block][3][2][nb][nb], added in block order.  Bound by the FP64 MMAs and the
// barriers between the phases (two blocks per SM fill each other's): 65,536 points x 24 functions, 2 + 2
// electrons, 8.0 -> 2.6 ms against FP64 FMAs from shared memory on the complex layout (4.8 GB); the sums with run-time
// sizes took 3.4 ms (address arithmetic).
constexpr int kFusedMaxNb = kTensorPadNb;
constexpr int kFusedWaitCode = 60;
__host__ __device__ constexpr int fusedWarps(int ntb) { return ntb == 4 ? 16 : 8; }
// column tiles (5) or row tiles (4) a warp accumulates
__host__ __device__ constexpr int fusedElemTiles(int ntb) { return ntb == 1 ? 1 : (ntb == 2 ? 5 : (ntb == 3 ? 19 : 9)); }

__device__ __forceinline__ double2 zfma(double2 a, double2 b, double2 c)   // a b + c
{
  return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ double2 zcfma(double2 a, double2 b, double2 c)  // conj(a) b + c
{
  return make_double2(fma(a.x, b.x, fma(a.y, b.y, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
}

// Shared-memory layout of kTcFused in doubles.  NB: the basis size rounded up to 4, the planes' row stride; every vector is
// padded to it with zeros, so that the loops and offsets are constants.  What depends on the electron counts comes last
template <int NB>
struct FusedLayout {
  static constexpr int NTB = (NB + 7) / 8, NW = fusedWarps(NTB), PS = tensorPlane(NB), NS = 8 * NTB + 4;   // NS: complex per slot, two slots on different banks
  static constexpr int planes = 0;                            // and zeros: fragments past a plane's last rows
  static constexpr int D = planes + 8 * PS + 4 * 32 + 16;     // {D0, D1}(i, j) at 4 (i NB + j), zeros behind
  static constexpr int X0 = D + 4 * (PS + 4);                 // {kv0, kv1, kc0, kc1} per row
  static constexpr int KG = X0 + NB * 12 + 8;                 // {kg0, kg1} per component and row
  static constexpr int EL = KG + 3 * (NB * 4 + 8);            // {ell0, ell1}
  static constexpr int Pw = EL + 3 * (NB * 4 + 8);
  static constexpr int Fai = Pw + 4 * NS;
  static constexpr int vai = Fai + 4 * NB;                    // [spin][component][i]
  static constexpr int SVD = vai + 12 * NB;
  static constexpr int tp = SVD + 4 * NB;                     // trace partials [warp][plane][8]
  static constexpr int tr = tp + NW * 64;                     // traces [plane][D0, D1]
  static constexpr int sc = tr + 32;                          // per spin: SG[3], SCV[3], occ, sumN (same, opposite)
  static constexpr int W = sc + 40;
  static constexpr int g = W + 96;
  static constexpr int v = g + 6 * NB;
  static constexpr int slot = v + NB;
  // per spin 16 + 6 max(nel) slots of NS complex: A 0..5, B 6..11, then the shared ones (VTs, Vjb, a zero); the occupied orbitals
  // [NB][ldc], spin 0's columns then spin 1's, ldc = 4 mod 8
  static int spinStride(int nel0, int nel1) { return 2 * NS * (16 + 6 * std::max(nel0, nel1)); }
  static int ldc(int nel0, int nel1) { return (2 * (nel0 + nel1) + 7) / 8 * 8 + 4; }
  static int total(int nel0, int nel1) { return slot + 2 * spinStride(nel0, nel1) + NB * ldc(nel0, nel1); }
  static size_t bytes(int nel0, int nel1) { return size_t(total(nel0, nel1)) * sizeof(double) + 32; }   // + mbarrier, abort word
};

struct TcFusedArgs {
  int64_t n1;
  int nb, nel[2];
  int spinStride, ldc, CB, total;   // FusedLayout
  const double * Fs;        // [n1][ps]
  const double * Fo;
  const double * Vs;        // [n1][3][ps]
  const double * Vo;
  const double * phi;       // [n1][nb]
  const double2 * grads;    // [n1][nb][3], reference basis
  const double * w;
  const DevSto * sto;
  const double2 * D;        // [2][nb][nb], real-harmonic basis
  const double2 * C0;       // occupied orbitals [nel][nb], reference basis
  const double2 * C1;
  double2 * part;           // [gridDim.x][3][2][nb][nb]
  int * status;
};

template <int NB>
__global__ void __launch_bounds__(32 * FusedLayout<NB>::NW, FusedLayout<NB>::NTB == 4 ? 1 : 2) kTcFused(const __grid_constant__ TcFusedArgs t)
{
  using L = FusedLayout<NB>;
  constexpr int NTB = L::NTB, NW = L::NW, PS = L::PS, NS = L::NS, NTH = 32 * NW, ET = fusedElemTiles(NTB), NACC = 6 * NTB > ET ? 6 * NTB : ET;
  extern __shared__ __align__(16) double sm[];
  int const nb = t.nb, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fr = lane >> 2, fq = lane & 3;
  uint64_t * bar = reinterpret_cast<uint64_t *>(sm + t.total);
  int * abortWord = reinterpret_cast<int *>(bar + 1);
  double2 const zero = make_double2(0, 0);
  auto z2 = [&](int o) -> double2 & { return *reinterpret_cast<double2 *>(sm + o); };
  // complex entry i of a slot of spin s: A 0..5, B 6..11, shared 12.. (VTs 12 + c, Vjb 15 + (t nel + b) 3 + c)
  auto slotAt = [&](int s, int k, int i) { return L::slot + s * t.spinStride + 2 * (k * NS + i); };

  for (int e = tid; e < t.total; e += NTH) sm[e] = 0.0;
  __syncthreads();
  for (int e = tid; e < 2 * nb * nb; e += NTH) {
    int const s = e / (nb * nb), r = e - s * nb * nb;
    z2(L::D + 4 * (r / nb * NB + r % nb) + 2 * s) = t.D[e];
  }
  for (int e = tid; e < (t.nel[0] + t.nel[1]) * nb; e += NTH) {
    // C_R(k, b) = sum_i conj(U[k][i]) C(i, b)
    int const m = e / nb, k = e % nb;
    const double2 * C = m < t.nel[0] ? t.C0 + m * nb : t.C1 + (m - t.nel[0]) * nb;
    double2 c = zmul(zconj(uRow(t.sto, k, k)), C[k]);
    if (t.sto[k].partner >= 0) c = zadd(c, zmul(zconj(uRow(t.sto, k, t.sto[k].partner)), C[t.sto[k].partner]));
    z2(t.CB + k * t.ldc + 2 * m) = c;
  }
  if (tid == 0) {
    tc::mbarInit(bar, 1);
    *abortWord = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc::fenceProxyAsync();   // the zeros above are written before the first copies land
  __syncthreads();
  constexpr uint32_t pB = uint32_t(PS) * 8u;
  auto issue = [&](int64_t p) {
    tc::mbarArriveTx(bar, 8u * pB + uint32_t(nb) * 48u);
    tc::bulkLoad(sm + L::planes, t.Vs + p * 3 * PS, 3 * pB, bar);
    tc::bulkLoad(sm + L::planes + 3 * PS, t.Vo + p * 3 * PS, 3 * pB, bar);
    tc::bulkLoad(sm + L::planes + 6 * PS, t.Fs + p * PS, pB, bar);
    tc::bulkLoad(sm + L::planes + 7 * PS, t.Fo + p * PS, pB, bar);
    tc::bulkLoad(sm + L::g, t.grads + p * nb * 3, uint32_t(nb) * 48u, bar);
  };
  int const G = gridDim.x;
  if (tid == 0 && blockIdx.x < t.n1) issue(blockIdx.x);

  // roles of the accumulating phases: warps 0 .. 2 NTB - 1 hold (spin, j tile) outer products, the others row tiles of (4)
  bool const outer = warp < 2 * NTB;
  int const os = warp / NTB, oj = 8 * (warp % NTB) + fr;
  constexpr int EW = NW - 2 * NTB;
  int const np = nb * (nb + 1) / 2, ew = warp - 2 * NTB;
  // offsets j NB + i of the upper-triangle elements this lane reads (row p of tile ew + q EW; rows past the last repeat it and
  // are not written), two per register
  uint32_t eoff[(ET + 1) / 2];
#pragma unroll
  for (int q = 0; q < ET; ++q) {
    int p = min((ew + q * EW) * 8 + fr, np - 1), j = 0;
    if (!outer)
      while (p >= nb - j) { p -= nb - j; ++j; }
    uint32_t const o = outer ? 0 : uint32_t(j * NB + j + p);
    if (q & 1) eoff[q / 2] |= o << 16;
    else eoff[q / 2] = o;
  }
  auto elem = [&](int q) { return int((eoff[q / 2] >> (q & 1 ? 16 : 0)) & 0xffffu); };
  double acc[NACC][2];
#pragma unroll
  for (int q = 0; q < NACC; ++q) acc[q][0] = acc[q][1] = 0.0;

  int k = 0;
  for (int64_t p = blockIdx.x; p < t.n1; p += G, ++k) {
    double const vnew = tid < nb ? t.phi[p * nb + tid] : 0.0;
    double const w = t.w[p];
    bool const ok = tc::waitBar(bar, uint32_t(k) & 1u, abortWord, t.status, kFusedWaitCode);
    if (tid < nb) {
      // v; as a complex slot entry it is A 0 and 4 and B 5 of both spins
      sm[L::v + tid] = vnew;
      for (int s = 0; s < 2; ++s) sm[slotAt(s, 0, tid)] = sm[slotAt(s, 4, tid)] = sm[slotAt(s, 11, tid)] = vnew;
    }
    if (__syncthreads_or(!ok)) return;
    const double2 * graw = reinterpret_cast<const double2 *>(sm + L::g);

    // phase 0: kv, kc per spin; gradients in the real-harmonic basis (B 1..3).  A warp per vector, lane = i
    for (int kind = warp; kind < 7; kind += NW) {
      int const i = lane;
      if (i >= nb) continue;
      if (kind < 2) {
        double2 a = zero;
        const double * d = sm + L::D + 4 * i + 2 * kind;
#pragma unroll
        for (int kk = 0; kk < NB; ++kk) a = zrfma(sm[L::v + kk], *reinterpret_cast<const double2 *>(d + 4 * kk * NB), a);
        z2(L::X0 + 12 * i + 2 * kind) = a;
      } else if (kind < 4) {
        double2 a = zero;
        const double * d = sm + L::D + 4 * i * NB + 2 * (kind - 2);
#pragma unroll 8
        for (int kk = 0; kk < NB; ++kk) {
          int l = kk + i;   // skewed: the lanes' rows of D fall on different banks
          l = l >= NB ? l - NB : l;
          a = zrfma(sm[L::v + l], *reinterpret_cast<const double2 *>(d + 4 * l), a);
        }
        z2(L::X0 + 12 * i + 4 + 2 * (kind - 2)) = a;
      } else {
        int const c = kind - 4, q = t.sto[i].partner;
        double2 gr = zmul(uRow(t.sto, i, i), graw[3 * i + c]);
        if (q >= 0) gr = zadd(gr, zmul(uRow(t.sto, i, q), graw[3 * q + c]));
        z2(slotAt(0, 7 + c, i)) = gr;
        z2(slotAt(1, 7 + c, i)) = gr;
      }
    }
    __syncthreads();
    // phase 1: kg per (spin, component), a warp each, lane = i
    for (int it = warp; it < 6; it += NW) {
      int const s = it / 3, c = it % 3;
      if (lane >= nb) continue;
      double2 a = zero;
      const double * d = sm + L::D + 4 * lane + 2 * s;
      const double * x = sm + slotAt(0, 7 + c, 0);
#pragma unroll
      for (int kk = 0; kk < NB; ++kk) a = zfma(*reinterpret_cast<const double2 *>(d + 4 * kk * NB), *reinterpret_cast<const double2 *>(x + 2 * kk), a);
      z2(L::KG + c * (NB * 4 + 8) + 4 * lane + 2 * s) = a;
    }
    __syncthreads();
    // phase 2: planes times vectors, one (plane, row tile) at a time, its fragments loaded once; then this warp's share of
    // the traces
    auto loadTile = [&](int plane, int jt, double (&A)[NB / 4]) {
      const double * x = sm + L::planes + plane * PS + 8 * jt + fr + fq * NB;
#pragma unroll
      for (int u = 0; u < NB / 4; ++u) A[u] = x[4 * u * NB];
    };
    auto rowTile = [&](double const (&A)[NB / 4], int b, int ldb, double (&d)[2]) {
      const double * x = sm + b + fq * ldb + fr;
#pragma unroll
      for (int u = 0; u < NB / 4; ++u) dmma(d, A[u], x[4 * u * ldb]);
    };
    for (int it = warp; it < 7 * NTB; it += NW) {
      int const plane = it / NTB, jt = it % NTB, j = 8 * jt + fr;   // Vs 0..2, Vo 3..5, Fs 6: the costly ones first
      bool const in = j < nb;
      double A[NB / 4];
      loadTile(plane, jt, A);
      if (plane < 3) {
        double d[2] = {0, 0}, e[2] = {0, 0};
        rowTile(A, L::X0, 12, d);
        rowTile(A, L::KG + plane * (NB * 4 + 8), 4, e);
        if (in) {
          // columns kv0, kv1: V-tilde_i of both spins; kc0, kc1: Vja
          z2(fq < 2 ? slotAt(fq, 12 + plane, j) : slotAt(fq - 2, 1 + plane, j)) = make_double2(d[0], d[1]);
          if (fq < 2) z2(L::vai + 2 * ((fq * 3 + plane) * NB + j)) = make_double2(e[0], e[1]);
        }
      } else if (plane == 6) {
        double d[2] = {0, 0};
        rowTile(A, L::X0, 12, d);
        if (in && fq < 2) z2(L::Fai + 2 * (fq * NB + j)) = make_double2(d[0], d[1]);
      }
      if (plane < 6)
        for (int n = 0; 8 * n + 4 < t.ldc; ++n) {
          double d[2] = {0, 0};
          rowTile(A, t.CB + 8 * n, t.ldc, d);
          int const m = 4 * n + fq, s = m < t.nel[0] ? 0 : 1, b = s ? m - t.nel[0] : m;
          if (in && m < t.nel[0] + t.nel[1]) z2(slotAt(s, 15 + (plane / 3 * t.nel[s] + b) * 3 + plane % 3, j)) = make_double2(d[0], d[1]);
        }
    }
    {
      double d[3][2] = {};
      const double * A = sm + L::planes + fr * PS + fq + 4 * warp;
      const double * B = sm + L::D + 4 * (fq + 4 * warp) + fr;
      constexpr int KS = NB * NB / 4, EACH = (KS + NW - 1) / NW;
#pragma unroll
      for (int u = 0; u < EACH; ++u)
        if ((u + 1) * NW <= KS || u * NW + warp < KS) dmma(d[u % 3], A[4 * NW * u], B[16 * NW * u]);
      z2(L::tp + 64 * warp + 8 * fr + 2 * fq) = make_double2(d[0][0] + d[1][0] + d[2][0], d[0][1] + d[1][1] + d[2][1]);
    }
    __syncthreads();
    // phase 3, a warp per item: ell per (spin, component), lane = k; sumN = sum_ab |sum_j conj(C(j,a)) Vjb(j,b)|^2 per (spin, tensor);
    // SG and occ; SCV per spin; the traces
    for (int it = warp; it < 14; it += NW) {
      if (it < 6) {
        int const s = it / 3, c = it % 3;
        if (lane < nb) {
          double2 a = zero;
          const double * d = sm + L::D + 4 * lane + 2 * s;
          const double * x = sm + slotAt(s, 12 + c, 0);
#pragma unroll
          for (int l = 0; l < NB; ++l) a = zfma(*reinterpret_cast<const double2 *>(d + 4 * l * NB), *reinterpret_cast<const double2 *>(x + 2 * l), a);
          z2(L::EL + c * (NB * 4 + 8) + 4 * lane + 2 * s) = a;
        }
      } else if (it < 10) {
        // rows: re and im of 4 orbitals a; columns: re and im of 4 of the 3 nel vectors Vjb(b, c)
        int const s = (it - 6) >> 1, tt = (it - 6) & 1, ne = t.nel[s];
        double sum = 0;
        for (int a0 = 0; a0 < ne; a0 += 4)
          for (int q0 = 0; q0 < 3 * ne; q0 += 4) {
            double d[2] = {0, 0};
            const double * A = sm + t.CB + 2 * ((s ? t.nel[0] : 0) + a0) + fr + fq * t.ldc;
            const double * B = sm + slotAt(s, 15 + tt * 3 * ne + q0, 0) + (fr >> 1) * 2 * NS + (fr & 1) + 2 * fq;
            bool const aIn = a0 + (fr >> 1) < ne, qIn = q0 + (fr >> 1) < 3 * ne;
#pragma unroll
            for (int u = 0; u < NB / 4; ++u) dmma(d, aIn ? A[4 * u * t.ldc] : 0.0, qIn ? B[8 * u] : 0.0);
            // rows 2 a (C.re) and 2 a + 1 (C.im), this lane's column pair (V.re, V.im)
            double const x = __shfl_down_sync(0xffffffffu, d[0], 4), y = __shfl_down_sync(0xffffffffu, d[1], 4);
            double const re = d[0] + y, im = d[1] - x;
            if (!(fr & 1)) sum += re * re + im * im;
          }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) sm[L::sc + 20 * s + 14 + tt] = sum;
      } else if (it < 13) {
        // rows: kv0, kv1, kc0, kc1 (re, im); columns: the three components of g and v, or of VTs_s (re, im)
        int const s = it - 11;   // -1: g
        double d[2] = {0, 0};
        const double * A = sm + L::X0 + 12 * fq + fr;
        const double * B = fr < 6 ? sm + slotAt(s < 0 ? 0 : s, (s < 0 ? 7 : 12) + (fr >> 1), 0) + (fr & 1) + 2 * fq : sm + L::v + fq;
        int const bs = fr < 6 ? 2 : 1;
#pragma unroll
        for (int u = 0; u < NB / 4; ++u) dmma(d, A[48 * u], fr == 7 ? 0.0 : B[4 * u * bs]);
        double const x = __shfl_down_sync(0xffffffffu, d[0], 4), y = __shfl_down_sync(0xffffffffu, d[1], 4);
        if (s < 0) {
          if (fq < 3 && (fr == 4 || fr == 6)) z2(L::sc + 20 * ((fr - 4) >> 1) + 2 * fq) = make_double2(d[0] - y, d[1] + x);   // SG = kc g
          if (fq == 3 && (fr == 0 || fr == 2)) sm[L::sc + 20 * (fr >> 1) + 12] = d[0];                                    // occ = Re kv v
        } else if (fq < 3 && fr == 2 * s) z2(L::sc + 20 * s + 2 * (3 + fq)) = make_double2(d[0] + y, x - d[1]);              // SCV = conj(VTs) kv
      } else {
        double a = 0;
        for (int u = 0; u < NW; ++u) a += sm[L::tp + 64 * u + 8 * (lane / 4) + lane % 4];
        sm[L::tr + lane] = a;
      }
    }
    __syncthreads();
    // phase 4: V ell (the first warps); the weights of the terms linear in the planes (the last warp)
    auto trace = [&](int plane, int s) { return z2(L::tr + 4 * plane + 2 * s); };
    if (warp < NTB) {
      double d[3][2] = {};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double A[NB / 4];
        loadTile(c, warp, A);
        rowTile(A, L::EL + c * (NB * 4 + 8), 4, d[c]);
      }
      int const j = 8 * warp + fr;
      if (j < nb && fq < 2) z2(L::SVD + 2 * (fq * NB + j)) = make_double2(d[0][0] + d[1][0] + d[2][0], d[0][1] + d[1][1] + d[2][1]);
    } else if (warp == NW - 1 && lane < 24) {
      // W[plane][spin, vector / three, re / im] at 12 plane + 4 spin + 2 kind
      int const plane = lane >> 2, s = (lane >> 1) & 1, kind = lane & 1, c = plane % 3, u = plane < 3 ? s : 1 - s;
      double2 x = z2(L::sc + 20 * u + 2 * c);
      if (kind) {
        double2 const vt = zadd(trace(c, u), trace(3 + c, 1 - u)), scv = z2(L::sc + 20 * u + 2 * (3 + c));
        double const oc = sm[L::sc + 20 * u + 12];
        x = make_double2(2.0 * oc * vt.x - 2.0 * scv.x, 2.0 * oc * vt.y - 2.0 * scv.y);
      }
      z2(L::W + 12 * plane + 4 * s + 2 * kind) = zscale(w, x);
    }
    __syncthreads();
    // phase 5: the vectors of the outer products (the outer-product warps); the terms linear in the planes (the others)
    if (outer) {
      for (int it = warp; it < 8; it += 2 * NTB) {
        int const kind = it >> 1, s = it & 1, i = lane, u = 1 - s;
        if (i >= nb) continue;
        double const vi = sm[L::v + i];
        double2 const svd = z2(L::SVD + 2 * (s * NB + i));
        double2 x = zero;
        if (kind == 0) {
          double2 const faa = zadd(trace(6, s), trace(7, u));
          x = zsub(zscale(vi, faa), z2(L::Fai + 2 * (s * NB + i)));
          z2(L::Pw + 2 * (s * NS + i)) = x;
          continue;
        }
        double nvt = 0;
        for (int c = 0; c < 3; ++c) {
          double2 const vt = zadd(trace(c, s), trace(3 + c, u)), vts = z2(slotAt(s, 12 + c, i));
          if (kind == 1) x = zsub(zfma(vt, z2(slotAt(0, 7 + c, i)), x), z2(L::vai + 2 * ((s * 3 + c) * NB + i)));
          else if (kind == 2) { x = zfma(vt, vts, x); nvt += vt.x * vt.x + vt.y * vt.y; }
          else x = zcfma(vts, vt, x);
        }
        if (kind == 1) z2(slotAt(s, 6, i)) = x;                                                  // B 0
        else if (kind == 2) {
          double const coef = nvt - sm[L::sc + 20 * s + 14] - sm[L::sc + 20 * u + 15];
          z2(slotAt(s, 10, i)) = zadd(make_double2(coef * vi, 0.0), zscale(2.0, zsub(svd, x)));   // B 4
        } else z2(slotAt(s, 5, i)) = zsub(zconj(svd), x);                                        // A 5
      }
    } else {
      double const b0 = sm[L::W + 12 * fq + fr], b1 = sm[L::W + 12 * (4 + fq) + fr];
      const double * A = sm + L::planes + fq * PS;
#pragma unroll
      for (int q = 0; q < ET; ++q) {
        dmma(acc[q], A[elem(q)], b0);
        dmma(acc[q], A[4 * PS + elem(q)], b1);
      }
    }
    __syncthreads();
    // the planes and raw gradients are free: the next point's copies run under the outer products
    if (tid == 0 && p + G < t.n1) {
      tc::fenceProxyAsync();
      issue(p + G);
    }
    // phase 6: outer products.  k step u: terms 2 u + (fq >> 1), part fq & 1; offsets in doubles
    if (outer) {
      int const part = fq & 1, half = fq >> 1, ne = t.nel[os];
      double const occS = sm[L::sc + 20 * os + 12], occO = sm[L::sc + 20 * (1 - os) + 12];
      auto step = [&](int o, int a, int b, double fre, double fim) {
        double const x = sm[a], xr = fre * x, xi = fim * x;
#pragma unroll
        for (int n = 0; n < NTB; ++n) {
          dmma(acc[(2 * o) * NTB + n], xr, sm[b + 16 * n + part]);
          dmma(acc[(2 * o + 1) * NTB + n], xi, sm[b + 16 * n + 1 - part]);
        }
      };
      int const aj = slotAt(os, 0, oj) + part, bi = slotAt(os, 6, fr), term = 2 * NS;
      double const sgn = part ? -1.0 : 1.0;   // of the real part of a plain product
      step(0, aj, L::Pw + 2 * (os * NS + fr), half ? 0.0 : sgn * w, half ? 0.0 : w);            // scalar: v Pw
#pragma unroll
      for (int u = 0; u < 2; ++u) {                                                             // vector: v Qw, -Vja g
        double const f = u == 0 && half == 0 ? w : -w;
        step(1, aj + (2 * u + half) * term, bi + (2 * u + half) * term, sgn * f, f);
      }
      {                                                                                          // three: v Rw, 2 Tw v
        double const f = half ? 2.0 * w : w;
        step(2, aj + (4 + half) * term, bi + (4 + half) * term, sgn * f, f);
      }
      int const sj = slotAt(os, 12, oj) + part, si = slotAt(os, 12, fr), last = 3 + 6 * ne;
      for (int u = 0; u < last; u += 2) {
        // conj(VTs_j) VTs_i (a conjugated), Vjb_j conj(Vjb_i) (b conjugated), then the zero slot
        int const q = u + half;
        double const f = q < 3 ? 2.0 * w : (q < last ? -2.0 * w * (q < 3 + 3 * ne ? occS : occO) : 0.0);
        step(2, sj + q * term, si + q * term, f, (q < 3) == (part == 1) ? -f : f);
      }
    }
    // the next point's first writes (v in A 0, A 4, B 5) must not overtake phase 6
    __syncthreads();
  }

  // the sums linear in the planes to shared memory (both triangles), added by the warps that hold the outer products
  double * E = sm + L::planes;   // [8][PS], every copy has landed and been consumed
  if (!outer) {
#pragma unroll
    for (int q = 0; q < ET; ++q) {
      int const r = (ew + q * EW) * 8 + fr;
      if (r >= np) continue;
      int const j = elem(q) / NB, i = elem(q) % NB;
      for (int e = 0; e < 2; ++e) E[(2 * fq + e) * PS + j * NB + i] = E[(2 * fq + e) * PS + i * NB + j] = acc[q][e];
    }
  }
  __syncthreads();
  if (!outer || oj >= nb) return;
  int const nn = nb * nb;
  double2 * out = t.part + int64_t(blockIdx.x) * 6 * nn + os * nn + oj * nb;
#pragma unroll
  for (int n = 0; n < NTB; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      int const i = 8 * n + 2 * fq + e;
      if (i >= nb) continue;
      const double * x = E + 4 * os * PS + oj * NB + i;
      out[i] = make_double2(acc[n][e], acc[NTB + n][e]);
      out[2 * nn + i] = make_double2(acc[2 * NTB + n][e] + x[0], acc[3 * NTB + n][e] + x[PS]);
      out[4 * nn + i] = make_double2(acc[4 * NTB + n][e] + x[2 * PS], acc[5 * NTB + n][e] + x[3 * PS]);
    }
}

// out[e] = sum over blocks of part[block][e], e < n: 32 elements per block, 8 warps taking every eighth part each, added in warp order
__global__ void __launch_bounds__(256) kTcPartials(int nparts, int n, const double2 * part, double2 * out)
{
  __shared__ double2 red[8][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  double2 a = make_double2(0, 0);
  if (e < n)
#pragma unroll 4
    for (int b = warp; b < nparts; b += 8) a = zadd(a, part[int64_t(b) * n + e]);
  red[warp][lane] = a;
  __syncthreads();
  if (warp != 0 || e >= n) return;
  for (int k = 1; k < 8; ++k) a = zadd(a, red[k][lane]);
  out[e] = a;
}

// C_R(k, b) = sum_i conj(U[k][i]) C(i, b) of the occupied orbitals, stored (i, b) at [b nb + i]: n0 of them at C0, the rest at C1
__global__ void kOrbitalsToReal(int n0, int n, int nb, const DevSto * sto, const double2 * C0, const double2 * C1, double2 * CR)
{
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * nb; e += gridDim.x * blockDim.x) {
    int const b = e / nb, k = e % nb, q = sto[k].partner;
    const double2 * C = b < n0 ? C0 + b * nb : C1 + (b - n0) * nb;
    double2 c = zmul(zconj(uRow(sto, k, k)), C[k]);
    if (q >= 0) c = zadd(c, zmul(zconj(uRow(sto, k, q)), C[q]));
    CR[e] = c;
  }
}

// g_R(r, k) = sum_i U[k][i] g(r, i) of the basis gradients [rows][nb][3]
__global__ void kGradsToReal(int64_t rows, int nb, const DevSto * sto, const double2 * g, double2 * gR)
{
  TC_GRID_LOOP(rows * nb * 3)
  {
    int const k = int(idx / 3 % nb), q = sto[k].partner;
    double2 a = zmul(uRow(sto, k, k), g[idx]);
    if (q >= 0) a = zadd(a, zmul(uRow(sto, k, q), g[idx + 3 * (q - k)]));
    gR[idx] = a;
  }
}

// X(j,i) = sum_{k,l} U[k][j] XR(k,l) conj(U[l][i]) of `count` complex matrices
__global__ void kSumsToReference(int count, int nb, const DevSto * s, const double2 * XR, double2 * X)
{
  int const nn = nb * nb;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < count * nn; idx += gridDim.x * blockDim.x) {
    int const m = idx / nn, j = idx % nn / nb, i = idx % nb;
    int const kj[2] = {j, s[j].partner}, li[2] = {i, s[i].partner};
    double2 acc = make_double2(0, 0);
    for (int a = 0; a < 2; ++a)
      for (int b = 0; b < 2; ++b)
        if (kj[a] >= 0 && li[b] >= 0)
          acc = zadd(acc, zmul(zmul(uRow(s, kj[a], j), XR[m * nn + kj[a] * nb + li[b]]), zconj(uRow(s, li[b], i))));
    X[idx] = acc;
  }
}

// bytes of shared memory, or the launch, of kTcFused for this basis size
template <int NB>
int launchFused(tcscf_ctx * ctx, TcFusedArgs a, int grid)
{
  using L = FusedLayout<NB>;
  a.spinStride = L::spinStride(a.nel[0], a.nel[1]);
  a.ldc = L::ldc(a.nel[0], a.nel[1]);
  a.CB = L::slot + 2 * a.spinStride;
  a.total = L::total(a.nel[0], a.nel[1]);
  size_t const smem = L::bytes(a.nel[0], a.nel[1]);
  TCSCF_CUDA(ctx, cudaFuncSetAttribute(kTcFused<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  kTcFused<NB><<<grid, 32 * L::NW, smem, ctx->stream>>>(a);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}
template <class F>
auto fusedDispatch(int nb, F && f)
{
  switch ((nb + 3) / 4) {
    case 1: return f(std::integral_constant<int, 4>{});
    case 2: return f(std::integral_constant<int, 8>{});
    case 3: return f(std::integral_constant<int, 12>{});
    case 4: return f(std::integral_constant<int, 16>{});
    case 5: return f(std::integral_constant<int, 20>{});
    case 6: return f(std::integral_constant<int, 24>{});
    case 7: return f(std::integral_constant<int, 28>{});
    default: return f(std::integral_constant<int, 32>{});
  }
}

Tensor const * findTensor(tcscf_ctx * ctx, int id)
{
  auto it = ctx->tensors.find(id);
  return it == ctx->tensors.end() ? nullptr : &it->second;
}


struct TcInputs {
  Grid * g1 = nullptr;
  Tensor const * F[2] = {nullptr, nullptr};   // same, opposite
  Tensor const * V[2] = {nullptr, nullptr};
};

int checkTcInputs(tcscf_ctx * ctx, int r1, int fs, int fo, int vs, int vo, int nup, int ndown, TcInputs & in)
{
  in.g1 = findGrid(ctx, r1);
  TCSCF_CHECK(ctx, in.g1 && in.g1->nb > 0 && in.g1->ndim == 3, TCSCF_ERR_INVALID_ARGUMENT, "r1 grid needs a 3-D basis");
  TCSCF_CHECK(ctx, in.g1->grads, TCSCF_ERR_INVALID_ARGUMENT, "the TC build needs the r1 basis gradients");
  int const ids[4] = {fs, fo, vs, vo};
  for (int k = 0; k < 4; ++k) {
    Tensor const * t = findTensor(ctx, ids[k]);
    TCSCF_CHECK(ctx, t, TCSCF_ERR_INVALID_ARGUMENT, "unknown tensor handle");
    TCSCF_CHECK(ctx, t->n1 == in.g1->n && t->nb == in.g1->nb, TCSCF_ERR_INVALID_ARGUMENT, "tensor does not match the r1 grid");
    TCSCF_CHECK(ctx, (k < 2) == !t->vec, TCSCF_ERR_INVALID_ARGUMENT, "expected Fji (computeF) then Vji (computeV) handles");
    if (k < 2) in.F[k] = t; else in.V[k - 2] = t;
  }
  TCSCF_CHECK(ctx, in.F[0]->isComplex == in.F[1]->isComplex, TCSCF_ERR_INVALID_ARGUMENT, "both Fji must come from the same r2 grid kind");
  TCSCF_CHECK(ctx, nup >= 0 && ndown >= 0 && nup <= in.g1->nb && ndown <= in.g1->nb, TCSCF_ERR_INVALID_ARGUMENT, "bad electron counts");
  return TCSCF_OK;
}

// One TC Fock build on device buffers: D [2][nb][nb], C0 / C1 occupied orbitals, h real [nb][nb];
// outputs G2, G3, Fock [2][nb][nb] and the energy (device).  The fused kernel's status word is copied
// to *hostStatus (0: ok), which the caller reads after its next synchronisation.
int tcFockBuildDevice(tcscf_ctx * ctx, TcInputs const & in, int nup, int ndown, const double2 * dD, const double2 * dC0, const double2 * dC1,
                      const double * dH, int respectSym, double2 * dG2, double2 * dG3, double2 * dFock, double * dE, int * hostStatus)
{
  Grid const & g = *in.g1;
  int const nb = g.nb, nm = std::max(1, std::max(nup, ndown));
  int64_t const n1 = g.n;
  *hostStatus = 0;
  int const ntb = (nb + 7) / 8;
  size_t smem = 0;
  int optin = 0;
  if (nb <= kFusedMaxNb) {
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    smem = fusedDispatch(nb, [&](auto n) { return FusedLayout<decltype(n)::value>::bytes(nup, ndown); });
  }
  if (smem > 0 && smem <= size_t(optin)) {
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
    // two blocks per SM where shared memory allows (1 KB of each block's share is the system's)
    int const perSm = ntb < 4 && 2 * (smem + 1024) <= 228 * 1024 ? 2 : 1;
    int const grid = int(std::max<int64_t>(1, std::min<int64_t>(int64_t(sms) * perSm, n1)));
    size_t const nn = size_t(nb) * nb, nn6 = 6 * nn;
    void * p = nullptr;
    TCSCF_TRY(scratch(ctx, "tc_fused", sizeof(double2) * (nn6 * (size_t(grid) + 2) + 2 * nn) + 256, &p));
    double2 * part = static_cast<double2 *>(p);
    double2 * sumsR = part + nn6 * grid;
    double2 * sums = sumsR + nn6;
    double2 * DR = sums + nn6;
    int * dStatus = reinterpret_cast<int *>(DR + 2 * nn);
    TCSCF_CUDA(ctx, cudaMemsetAsync(dStatus, 0, sizeof(int), ctx->stream));
    for (int s = 0; s < 2; ++s) TCSCF_TRY(densityToRealLaunch(ctx, nb, g.dsto, dD + s * nn, DR + s * nn));
    TcFusedArgs a{};
    a.n1 = n1; a.nb = nb;
    a.nel[0] = nup; a.nel[1] = ndown;
    a.Fs = in.F[0]->d; a.Fo = in.F[1]->d; a.Vs = in.V[0]->d; a.Vo = in.V[1]->d;
    a.phi = g.phiR; a.grads = reinterpret_cast<const double2 *>(g.grads); a.w = g.w; a.sto = g.dsto;
    a.D = DR; a.C0 = dC0; a.C1 = dC1;
    a.part = part; a.status = dStatus;
    TCSCF_TRY(fusedDispatch(nb, [&](auto n) { return launchFused<decltype(n)::value>(ctx, a, grid); }));
    kTcPartials<<<unsigned((nn6 + 31) / 32), 256, 0, ctx->stream>>>(grid, int(nn6), part, sumsR);
    TCSCF_LAUNCH(ctx);
    kSumsToReference<<<gridBlocks(int64_t(nn6), 256), 256, 0, ctx->stream>>>(6, nb, g.dsto, sumsR, sums);
    TCSCF_LAUNCH(ctx);
    kTcAssemble<<<gridBlocks(2 * nb * nb, 256), 256, 0, ctx->stream>>>(nb, sums, dH, respectSym, dG2, dG3);
    TCSCF_LAUNCH(ctx);
    TCSCF_TRY(finalizeLaunch(ctx, 2, nb, dH, dG2, dG3, dD, respectSym, 1.0, dFock, dE));
    TCSCF_CUDA(ctx, cudaMemcpyAsync(hostStatus, dStatus, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    return TCSCF_OK;
  }
  // larger bases (or electron counts): the per-intermediate kernels on the same planes, over all points at once so that
  // kernels with a thread or warp per point fill the machine; in chunks only where the intermediates do not fit
  // the device beside the tensors.  Planes read in place, against expanding them to the complex layout in chunks of 1 GiB: 65,536 points,
  // 2 + 2 electrons: 138 -> 84 ms at 40 functions, 562 -> 274 ms at 64 (16,384 points 36.9 -> 21.0 and 140 -> 66 ms)
  size_t const nn = size_t(nb) * nb;
  size_t const perPoint = 1 + nb + 3 + 3 + nb + 3 * nb + 3 * nb + 2 * 3 * size_t(nb) * nm + nb + 3;   // double2 units
  int64_t chunk = n1;
  void * p = nullptr;
  size_t bytes = 0;
  for (int st = TCSCF_ERR_CUDA; st != TCSCF_OK;) {
    size_t const chunks = size_t((n1 + chunk - 1) / chunk);
    bytes = sizeof(double2) * (2 * size_t(chunk) * perPoint + size_t(chunk) * nb * 3 + 6 * nn * (chunks + 2) + 2 * nn + size_t(nup + ndown) * nb) +
            sizeof(double) * 2 * 3 * size_t(chunk) + 1024;
    st = scratch(ctx, "tc_terms", bytes, &p);
    if (st == TCSCF_OK) break;
    cudaGetLastError();   // the failed allocation is not the next launch's error
    if (chunk <= 1024) return st;
    chunk = (chunk + 1) / 2;
  }
  int const chunks = int((n1 + chunk - 1) / chunk);
  double2 * z = static_cast<double2 *>(p);
  auto take = [&](size_t n) { double2 * r = z; z += n; return r; };
  size_t const n2 = 2 * size_t(chunk);
  TcView t{};
  t.nb = nb; t.nelMax = nm; t.nel[0] = nup; t.nel[1] = ndown;
  t.ld = tensorStride(nb); t.ps = tensorPlane(nb);
  double2 * DR = take(2 * nn);
  double2 * C0 = take(size_t(nup) * nb);
  double2 * C1 = take(size_t(ndown) * nb);
  double2 * grads = take(size_t(chunk) * nb * 3);
  t.D = DR; t.C0 = C0; t.C1 = C1; t.grads = grads;
  t.Faa = take(n2); t.Fai = take(n2 * nb); t.VT = take(n2 * 3); t.SG = take(n2 * 3);
  t.Vai = take(n2 * nb); t.Vja = take(n2 * nb * 3); t.VTs = take(n2 * nb * 3);
  t.Vjbs = take(n2 * nb * nm * 3); t.Vjbo = take(n2 * nb * nm * 3); t.SVD = take(n2 * nb); t.SCV = take(n2 * 3);
  double2 * sums = take(6 * nn);
  double2 * sumsR = take(6 * nn);
  double2 * part = take(6 * nn * chunks);
  double * dr = reinterpret_cast<double *>(z);
  t.occD = dr; t.sumNs = dr + n2; t.sumNo = dr + 2 * n2;
  TCSCF_CHECK(ctx, reinterpret_cast<char *>(dr + 3 * n2) <= static_cast<char *>(p) + bytes, TCSCF_ERR_INVALID_ARGUMENT, "internal: tc scratch");
  for (int s = 0; s < 2; ++s) TCSCF_TRY(densityToRealLaunch(ctx, nb, g.dsto, dD + s * nn, DR + s * nn));
  kOrbitalsToReal<<<gridBlocks(int64_t(nup + ndown) * nb, 256), 256, 0, ctx->stream>>>(nup, nup + ndown, nb, g.dsto, dC0, dC1, C0);
  TCSCF_LAUNCH(ctx);
  for (int c = 0; c < chunks; ++c) {
    int64_t const r0 = c * chunk, rows = std::min(chunk, n1 - r0);
    t.n1 = rows;
    t.Fs = in.F[0]->d + r0 * t.ps; t.Fo = in.F[1]->d + r0 * t.ps;
    t.Vs = in.V[0]->d + 3 * r0 * t.ps; t.Vo = in.V[1]->d + 3 * r0 * t.ps;
    t.vals = g.phiR + r0 * nb;
    t.w = g.w + r0;
    kGradsToReal<<<gridBlocks(rows * nb * 3, 256), 256, 0, ctx->stream>>>(rows, nb, g.dsto, reinterpret_cast<const double2 *>(g.grads) + r0 * nb * 3, grads);
    TCSCF_LAUNCH(ctx);
    kTcPoint<<<gridBlocks(32 * rows, 128), 128, 0, ctx->stream>>>(t);
    TCSCF_LAUNCH(ctx);
    kTcPointI<<<gridBlocks(2 * rows * nb, 128), 128, 0, ctx->stream>>>(t);
    TCSCF_LAUNCH(ctx);
    kTcVjb<<<gridBlocks(2 * rows * nb * nm, 128), 128, 0, ctx->stream>>>(t);
    TCSCF_LAUNCH(ctx);
    kTcVab<<<gridBlocks(2 * rows, 128), 128, 0, ctx->stream>>>(t);
    TCSCF_LAUNCH(ctx);
    kTcSvd<<<gridBlocks(2 * rows * nb, 128), 128, 0, ctx->stream>>>(t);
    TCSCF_LAUNCH(ctx);
    kTcReduce<<<unsigned(2 * nb * nb), 256, 0, ctx->stream>>>(t, chunks == 1 ? sumsR : part + 6 * nn * c);
    TCSCF_LAUNCH(ctx);
  }
  if (chunks > 1) {
    kTcPartials<<<unsigned((6 * nn + 31) / 32), 256, 0, ctx->stream>>>(chunks, int(6 * nn), part, sumsR);
    TCSCF_LAUNCH(ctx);
  }
  kSumsToReference<<<gridBlocks(int64_t(6 * nn), 256), 256, 0, ctx->stream>>>(6, nb, g.dsto, sumsR, sums);
  TCSCF_LAUNCH(ctx);
  kTcAssemble<<<gridBlocks(2 * nb * nb, 256), 256, 0, ctx->stream>>>(nb, sums, dH, respectSym, dG2, dG3);
  TCSCF_LAUNCH(ctx);
  return finalizeLaunch(ctx, 2, nb, dH, dG2, dG3, dD, respectSym, 1.0, dFock, dE);
}

// S-metric modified Gram-Schmidt of orthogonalization.hpp:136-154 on nvec row vectors of length n,
// metric S real symmetric [n][n]; after the first vector the normalisation is Euclidean (:152).
void mgsMetric(std::vector<std::complex<double>> & v, int nvec, int n, std::vector<double> const & S)
{
  using cplx = std::complex<double>;
  auto ip = [&](cplx const * a, cplx const * b) {
    cplx d = 0;
    for (int i = 0; i < n; ++i) {
      cplx row = 0;
      for (int j = 0; j < n; ++j) row += S[size_t(i) * n + j] * b[j];
      d += std::conj(a[i]) * row;
    }
    return d;
  };
  auto normE = [&](cplx const * a) { double d = 0; for (int i = 0; i < n; ++i) d += std::norm(a[i]); return std::sqrt(d); };
  if (nvec == 0) return;
  double const s0 = 1.0 / std::sqrt(ip(v.data(), v.data()).real());
  for (int i = 0; i < n; ++i) v[i] *= s0;
  for (int i = 1; i < nvec; ++i) {
    for (int j = i; j < nvec; ++j) {
      cplx const sc = ip(v.data() + size_t(i - 1) * n, v.data() + size_t(j) * n);
      for (int k = 0; k < n; ++k) v[size_t(j) * n + k] -= sc * v[size_t(i - 1) * n + k];
    }
    double const s = 1.0 / normE(v.data() + size_t(i) * n);
    for (int k = 0; k < n; ++k) v[size_t(i) * n + k] *= s;
  }
}

}  // namespace
}  // namespace tcscf

using namespace tcscf;

extern "C" {

int tcscf_tc_fock_build(tcscf_ctx * ctx, int r1, int fji_same, int fji_oppo, int vji_same, int vji_oppo, int n_up, int n_down,
                        const double * density, const double * occ_up, const double * occ_down, const double * h, int respect_symmetry,
                        double * G2, double * G3, double * fock, double * energy)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  TcInputs in;
  TCSCF_TRY(checkTcInputs(ctx, r1, fji_same, fji_oppo, vji_same, vji_oppo, n_up, n_down, in));
  TCSCF_CHECK(ctx, density && h, TCSCF_ERR_INVALID_ARGUMENT, "density and h are required");
  TCSCF_CHECK(ctx, (occ_up || n_up == 0) && (occ_down || n_down == 0), TCSCF_ERR_INVALID_ARGUMENT, "occupied orbitals are required");
  int const nb = in.g1->nb;
  size_t const nn = size_t(nb) * nb;
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "tc_io", sizeof(double2) * (nn * 2 * 4 + size_t(nb) * (n_up + n_down) + 2) + sizeof(double) * (nn + 2), &p));
  double2 * dD = static_cast<double2 *>(p);
  double2 * dG2 = dD + 2 * nn;
  double2 * dG3 = dG2 + 2 * nn;
  double2 * dF = dG3 + 2 * nn;
  double2 * dC0 = dF + 2 * nn;
  double2 * dC1 = dC0 + size_t(nb) * n_up;
  double * dH = reinterpret_cast<double *>(dC1 + size_t(nb) * n_down + 1);
  double * dE = dH + nn;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dD, density, sizeof(double2) * 2 * nn, cudaMemcpyHostToDevice, ctx->stream));
  if (n_up) TCSCF_CUDA(ctx, cudaMemcpyAsync(dC0, occ_up, sizeof(double2) * nb * n_up, cudaMemcpyHostToDevice, ctx->stream));
  if (n_down) TCSCF_CUDA(ctx, cudaMemcpyAsync(dC1, occ_down, sizeof(double2) * nb * n_down, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dH, h, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  int kst = 0;
  TCSCF_TRY(tcFockBuildDevice(ctx, in, n_up, n_down, dD, dC0, dC1, dH, respect_symmetry, dG2, dG3, dF, dE, &kst));
  if (G2) TCSCF_CUDA(ctx, cudaMemcpyAsync(G2, dG2, sizeof(double2) * 2 * nn, cudaMemcpyDeviceToHost, ctx->stream));
  if (G3) TCSCF_CUDA(ctx, cudaMemcpyAsync(G3, dG3, sizeof(double2) * 2 * nn, cudaMemcpyDeviceToHost, ctx->stream));
  if (fock) TCSCF_CUDA(ctx, cudaMemcpyAsync(fock, dF, sizeof(double2) * 2 * nn, cudaMemcpyDeviceToHost, ctx->stream));
  double e = 0;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(&e, dE, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  TCSCF_CHECK(ctx, kst == 0, TCSCF_ERR_TIMEOUT, "TC build: bounded wait expired (code " + std::to_string(kst) + ")");
  if (energy) *energy = e;
  if (!(e == e) || std::isinf(e)) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite TC energy");
  return TCSCF_OK;
}

int tcscf_tc_scf(tcscf_ctx * ctx, int r1, int fji_same, int fji_oppo, int vji_same, int vji_oppo, const double * S, const double * h,
                 int n_up, int n_down, int respect_symmetry, double tol, int max_iter, double * energy, int * iterations, double * density,
                 double * pseudo_energies)
{
  TCSCF_NVTX();
  using cplx = std::complex<double>;
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  TcInputs in;
  TCSCF_TRY(checkTcInputs(ctx, r1, fji_same, fji_oppo, vji_same, vji_oppo, n_up, n_down, in));
  TCSCF_CHECK(ctx, S && h && energy && iterations && density, TCSCF_ERR_INVALID_ARGUMENT, "S, h and the outputs are required");
  TCSCF_CHECK(ctx, max_iter > 0, TCSCF_ERR_INVALID_ARGUMENT, "max_iter must be positive");
  int const nb = in.g1->nb;
  size_t const nn = size_t(nb) * nb;
  int const nel[2] = {n_up, n_down};
  cublasHandle_t blas = nullptr;
  TCSCF_TRY(blasHandle(ctx, &blas));
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "tc_scf", sizeof(double2) * (nn * 2 * 4 + size_t(nb) * (n_up + n_down) + 2 + 4 * nn + nb) + sizeof(double) * (2 * nn + 2) + 64,
                    &p));
  double2 * dD = static_cast<double2 *>(p);
  double2 * dG2 = dD + 2 * nn;
  double2 * dG3 = dG2 + 2 * nn;
  double2 * dF = dG3 + 2 * nn;
  double2 * dC0 = dF + 2 * nn;
  double2 * dC1 = dC0 + size_t(nb) * n_up;
  double2 * dA = dC1 + size_t(nb) * n_down + 1;
  double2 * dB = dA + nn;
  double2 * dVR = dB + nn;
  double2 * dVL = dVR + nn;
  double2 * dW = dVL + nn;
  double * dH = reinterpret_cast<double *>(dW + nb + 1);
  double * dS = dH + nn;
  double * dE = dS + nn;
  int * dInfo = reinterpret_cast<int *>(dE + 1);
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dH, h, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dS, S, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemsetAsync(dD, 0, sizeof(double2) * 2 * nn, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemsetAsync(dC0, 0, sizeof(double2) * (size_t(nb) * (n_up + n_down) + 1), ctx->stream));

  cusolverDnParams_t params = nullptr;
  TCSCF_CHECK(ctx, cusolverDnCreateParams(&params) == CUSOLVER_STATUS_SUCCESS, TCSCF_ERR_CUDA, "cusolverDnCreateParams failed");
  struct ParamsGuard { cusolverDnParams_t p; ~ParamsGuard() { cusolverDnDestroyParams(p); } } guard{params};
  size_t dws = 0, hws = 0;
  TCSCF_CHECK(ctx, cusolverDnXgeev_bufferSize(ctx->solver, params, CUSOLVER_EIG_MODE_NOVECTOR, CUSOLVER_EIG_MODE_VECTOR, nb, CUDA_C_64F, dA, nb,
                                              CUDA_C_64F, dW, CUDA_C_64F, dVL, nb, CUDA_C_64F, dVR, nb, CUDA_C_64F, &dws, &hws) == CUSOLVER_STATUS_SUCCESS,
              TCSCF_ERR_LINALG, "cusolverDnXgeev_bufferSize failed");
  int lpotrf = 0;
  TCSCF_CHECK(ctx, cusolverDnZpotrf_bufferSize(ctx->solver, CUBLAS_FILL_MODE_LOWER, nb, reinterpret_cast<cuDoubleComplex *>(dB), nb, &lpotrf) ==
                       CUSOLVER_STATUS_SUCCESS,
              TCSCF_ERR_LINALG, "cusolverDnZpotrf_bufferSize failed");
  void * wk = nullptr;
  TCSCF_TRY(scratch(ctx, "tc_scf_work", std::max(dws, sizeof(double2) * size_t(lpotrf)) + 256, &wk));
  std::vector<char> hwork(hws + 1);

  std::vector<int> sorted(2 * size_t(nb));
  for (int s = 0; s < 2; ++s)
    for (int i = 0; i < nb; ++i) sorted[size_t(s) * nb + i] = i;
  std::vector<cplx> hW(nb), hV(nn), hD(2 * nn);
  std::vector<cplx> occ[2] = {std::vector<cplx>(size_t(nb) * n_up), std::vector<cplx>(size_t(nb) * n_down)};
  std::vector<double> hS(S, S + nn);
  double prev = std::numeric_limits<double>::max();
  cuDoubleComplex const one = make_cuDoubleComplex(1, 0);
  for (int it = 0; it < max_iter; ++it) {
    int kst = 0;
    TCSCF_TRY(tcFockBuildDevice(ctx, in, n_up, n_down, dD, dC0, dC1, dH, respect_symmetry, dG2, dG3, dF, dE, &kst));
    double e = 0;
    TCSCF_CUDA(ctx, cudaMemcpyAsync(&e, dE, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    TCSCF_CHECK(ctx, kst == 0, TCSCF_ERR_TIMEOUT, "TC build: bounded wait expired (code " + std::to_string(kst) + ")");
    *iterations = it + 1;
    TCSCF_CHECK(ctx, e == e && !std::isinf(e), TCSCF_ERR_NONFINITE, "non-finite TC energy");
    if (std::abs(e - prev) < tol) {
      *energy = e;
      TCSCF_CUDA(ctx, cudaMemcpyAsync(density, dD, sizeof(double2) * 2 * nn, cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      return TCSCF_OK;
    }
    prev = e;
    for (int s = 0; s < 2; ++s) {
      // F C = S C e  ->  (L^-1 F L^-H) Y = Y e,  C = L^-H Y,  S = L L^H
      kToColMajorZ<<<gridBlocks(int64_t(nn), 256), 256, 0, ctx->stream>>>(nb, dF + s * nn, dA);
      TCSCF_LAUNCH(ctx);
      kRealToZ<<<gridBlocks(int64_t(nn), 256), 256, 0, ctx->stream>>>(int(nn), dS, dB);
      TCSCF_LAUNCH(ctx);
      auto * A = reinterpret_cast<cuDoubleComplex *>(dA);
      auto * B = reinterpret_cast<cuDoubleComplex *>(dB);
      auto * VR = reinterpret_cast<cuDoubleComplex *>(dVR);
      TCSCF_CHECK(ctx, cusolverDnZpotrf(ctx->solver, CUBLAS_FILL_MODE_LOWER, nb, B, nb, static_cast<cuDoubleComplex *>(wk), lpotrf, dInfo) ==
                           CUSOLVER_STATUS_SUCCESS,
                  TCSCF_ERR_LINALG, "cusolverDnZpotrf failed");
      int info = 0;
      TCSCF_CUDA(ctx, cudaMemcpyAsync(&info, dInfo, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      TCSCF_CHECK(ctx, info == 0, TCSCF_ERR_LINALG, "overlap matrix is not positive definite (potrf info " + std::to_string(info) + ")");
      TCSCF_CHECK(ctx, cublasZtrsm(blas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_N, CUBLAS_DIAG_NON_UNIT, nb, nb, &one, B, nb, A, nb) ==
                               CUBLAS_STATUS_SUCCESS &&
                           cublasZtrsm(blas, CUBLAS_SIDE_RIGHT, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_C, CUBLAS_DIAG_NON_UNIT, nb, nb, &one, B, nb, A, nb) ==
                               CUBLAS_STATUS_SUCCESS,
                  TCSCF_ERR_LINALG, "cublasZtrsm failed");
      TCSCF_CHECK(ctx, cusolverDnXgeev(ctx->solver, params, CUSOLVER_EIG_MODE_NOVECTOR, CUSOLVER_EIG_MODE_VECTOR, nb, CUDA_C_64F, dA, nb, CUDA_C_64F,
                                       dW, CUDA_C_64F, dVL, nb, CUDA_C_64F, dVR, nb, CUDA_C_64F, wk, dws, hwork.data(), hws, dInfo) ==
                           CUSOLVER_STATUS_SUCCESS,
                  TCSCF_ERR_LINALG, "cusolverDnXgeev failed");
      TCSCF_CHECK(ctx, cublasZtrsm(blas, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_C, CUBLAS_DIAG_NON_UNIT, nb, nb, &one, B, nb, VR, nb) ==
                           CUBLAS_STATUS_SUCCESS,
                  TCSCF_ERR_LINALG, "cublasZtrsm failed");
      TCSCF_CUDA(ctx, cudaMemcpyAsync(&info, dInfo, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaMemcpyAsync(hW.data(), dW, sizeof(double2) * nb, cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaMemcpyAsync(hV.data(), dVR, sizeof(double2) * nn, cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      TCSCF_CHECK(ctx, info == 0, TCSCF_ERR_LINALG, "cusolverDnXgeev info " + std::to_string(info));
      // sort by real part, keeping the previous iteration's order as the starting permutation (:1298-1303)
      int * si = sorted.data() + size_t(s) * nb;
      std::sort(si, si + nb, [&](int a, int b) { return hW[a].real() < hW[b].real(); });
      std::vector<cplx> occT(size_t(nel[s]) * nb);
      for (int i = 0; i < nel[s]; ++i) {
        if (pseudo_energies) pseudo_energies[size_t(s) * nb + i] = hW[si[i]].real();
        for (int j = 0; j < nb; ++j) occT[size_t(i) * nb + j] = hV[size_t(si[i]) * nb + j];
      }
      mgsMetric(occT, nel[s], nb, hS);
      occ[s] = occT;   // column-major nb x nel: column b = row b of occT
      // getNewDensity (:20-44): D(u,v) = sum_a C(u,a) conj(C(v,a))
      for (int u = 0; u < nb; ++u)
        for (int v = 0; v < nb; ++v) {
          cplx t = 0;
          for (int a = 0; a < nel[s]; ++a) t += occT[size_t(a) * nb + u] * std::conj(occT[size_t(a) * nb + v]);
          hD[size_t(s) * nn + size_t(u) * nb + v] = t;
        }
    }
    TCSCF_CUDA(ctx, cudaMemcpyAsync(dD, hD.data(), sizeof(double2) * 2 * nn, cudaMemcpyHostToDevice, ctx->stream));
    if (n_up) TCSCF_CUDA(ctx, cudaMemcpyAsync(dC0, occ[0].data(), sizeof(double2) * nb * n_up, cudaMemcpyHostToDevice, ctx->stream));
    if (n_down) TCSCF_CUDA(ctx, cudaMemcpyAsync(dC1, occ[1].data(), sizeof(double2) * nb * n_down, cudaMemcpyHostToDevice, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));   // host buffers are reused next iteration
  }
  *energy = prev;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(density, dD, sizeof(double2) * 2 * nn, cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return fail(ctx, TCSCF_ERR_NOT_CONVERGED, "TC SCF did not converge in " + std::to_string(max_iter) + " iterations");
}

}  // extern "C"
