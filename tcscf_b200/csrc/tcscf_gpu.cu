// libtcscf_gpu.so: context, device grids and basis evaluation, one-electron quadrature, density
// factorisation, the Fock-build pipeline (direct and precompute forms) and the SCF driver.
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>
#include <string>
#include <algorithm>
#include <vector>

#include "kernels.cuh"

namespace tcscf {

int fail(tcscf_ctx * ctx, int code, std::string const & msg)
{
  if (ctx) ctx->err = msg;
  return code;
}

int blasHandle(tcscf_ctx * ctx, cublasHandle_t * out)
{
  if (!ctx->blas && cublasCreate(&ctx->blas) != CUBLAS_STATUS_SUCCESS) return fail(ctx, TCSCF_ERR_CUDA, "cublasCreate failed");
  if (cublasSetStream(ctx->blas, ctx->stream) != CUBLAS_STATUS_SUCCESS) return fail(ctx, TCSCF_ERR_CUDA, "cublasSetStream failed");
  *out = ctx->blas;
  return TCSCF_OK;
}

int scratch(tcscf_ctx * ctx, char const * name, size_t bytes, void ** out)
{
  Scratch & s = ctx->scratch[name];
  if (s.bytes < bytes || !s.p) {
    if (s.p) { cudaStreamSynchronize(ctx->stream); cudaFree(s.p); s.p = nullptr; s.bytes = 0; }
    size_t const want = std::max<size_t>(bytes, 256);
    cudaError_t const e = cudaMalloc(&s.p, want);
    if (e != cudaSuccess) return fail(ctx, TCSCF_ERR_CUDA, std::string("cudaMalloc(scratch ") + name + "): " + cudaGetErrorString(e));
    s.bytes = want;
  }
  *out = s.p;
  return TCSCF_OK;
}

Grid * findGrid(tcscf_ctx * ctx, int id)
{
  auto it = ctx->grids.find(id);
  return it == ctx->grids.end() ? nullptr : &it->second;
}

int gridAllocBytes(tcscf_ctx * ctx, void ** p, size_t bytes)
{
  *p = nullptr;
  cudaError_t const e = cudaMallocFromPoolAsync(p, std::max<size_t>(bytes, 256), ctx->gridPool, ctx->stream);
  if (e != cudaSuccess) return fail(ctx, TCSCF_ERR_CUDA, std::string("grid buffer allocation: ") + cudaGetErrorString(e));
  if (reinterpret_cast<uintptr_t>(*p) % 256 != 0) {
    cudaFreeAsync(*p, ctx->stream);
    *p = nullptr;
    return fail(ctx, TCSCF_ERR_CUDA, "grid buffer allocation is not 256-byte aligned");
  }
  return TCSCF_OK;
}

void gridRelease(tcscf_ctx * ctx, void * p)
{
  if (p) cudaFreeAsync(p, ctx->stream);
}

void gridReleaseAll(tcscf_ctx * ctx, Grid & g)
{
  gridRelease(ctx, g.pts); gridRelease(ctx, g.w); gridRelease(ctx, g.dsto); gridRelease(ctx, g.phiR);
  gridRelease(ctx, g.vals); gridRelease(ctx, g.grads); gridRelease(ctx, g.vtCache);
  g.pts = g.w = g.phiR = g.vals = g.grads = nullptr;
  g.dsto = nullptr;
  g.vtCache = nullptr;
}

namespace {

// Fully normalised associated Legendre function with the Condon-Shortley phase,
// P(l, m, cos t) = (-1)^m sqrt((2l+1)/(4 pi) (l-m)!/(l+m)!) P_l^m(cos t), i.e. Y_l^m(t, 0), evaluated
// with the standard three-term recurrences in l at fixed m (x = cos t, s = sin t).
__device__ double sphLegendre(int l, int m, double x, double s)
{
  if (m > l || m < 0) return 0.0;
  double pmm = 1.0;
  for (int k = 1; k <= m; ++k) pmm *= -s * sqrt((2.0 * k - 1.0) / (2.0 * k));
  pmm *= sqrt((2.0 * m + 1.0) / (4.0 * kPi));
  if (l == m) return pmm;
  double pm1 = x * sqrt(2.0 * m + 3.0) * pmm;
  if (l == m + 1) return pm1;
  double pll = 0.0;
  for (int ll = m + 2; ll <= l; ++ll) {
    double const a = sqrt((4.0 * ll * ll - 1.0) / (double(ll) * ll - double(m) * m));
    double const b = sqrt((double(ll - 1) * (ll - 1) - double(m) * m) / (4.0 * (ll - 1) * (ll - 1) - 1.0));
    pll = a * (x * pm1 - b * pmm);
    pmm = pm1;
    pm1 = pll;
  }
  return pll;
}

// QMCGrid::setBasisFunctions (integrateAll.hpp:88-137) with SlaterTypeOrbital::operator() and
// ::gradient (SlaterTypeOrbital.hpp:51-106), or the Ochi / hydrogen-like radial parts (basisRadial;
// OchiBasisFunction::gradient, OchiBasis.hpp:58-107, shares the angular terms of the STO gradient).  Also writes
// the real-harmonic values phiR used by the contraction kernels: cos-type sqrt2 R P cos(|m| phi) for m > 0,
// sin-type sqrt2 R P sin(|m| phi) for m < 0, R P for m == 0.
// A block takes `npts` points.  What depends on the point alone (angles, unit vectors, cos / sin of m phi, the associated
// Legendre functions of every l <= lmax) is formed once in shared memory; then one thread per (point,
// function), function index fastest so that every store is coalesced, has the radial part and products left.
// Bound by its stores and the FP64 exponentials.  With every thread forming the angles for itself: 59,000
// points x 40 functions with gradients 224 -> 57 us.
constexpr int kBasisHead = 12;   // doubles per point before the tables
__host__ __device__ inline int basisPointDoubles(int lmax) { return kBasisHead + 2 * (lmax + 2) + (lmax + 1) * (lmax + 2) / 2; }
__global__ void __launch_bounds__(256) kBasis(int64_t n, int nb, int ndim, int lmax, int npts, const double * __restrict__ pts,
                                            const DevSto * __restrict__ sto, double * __restrict__ phiR, double * __restrict__ vals,
                                            double * __restrict__ grads)
{
  extern __shared__ double sm[];
  int const per = basisPointDoubles(lmax), nm = lmax + 2, nlm = (lmax + 1) * (lmax + 2) / 2, tid = threadIdx.x;
  int64_t const i0 = int64_t(blockIdx.x) * npts;
  int const np = int(min(int64_t(npts), n - i0));
  // per point: r, cos and sin theta of the Legendre functions, phi (replaced below), then for the gradients 1/r, cot theta,
  // 1/(r sin theta) and the unit vectors' sines and cosines; cos, sin (m phi); P(l, m)
  for (int t = tid; t < np; t += 256) {
    double * q = sm + t * per;
    double const x = pts[i0 + t], y = pts[n + i0 + t], z = pts[2 * n + i0 + t];
    double const r = norm3d(x, y, z);
    q[0] = r;
    q[1] = z / r;
    q[2] = sqrt(x * x + y * y) / r;
    q[3] = atan2(y, x);
    if (grads) {
      double const th = acos(q[1]);
      double sth, cth;
      sincos(th, &sth, &cth);
      q[4] = 1.0 / r;
      q[5] = 1.0 / tan(th);
      q[6] = 1.0 / (r * sth);
      q[7] = sth;
      q[8] = cth;
    }
  }
  __syncthreads();
  for (int t = tid; t < np * (nm + nlm); t += 256) {
    int const k = t / np;
    double * q = sm + (t % np) * per;
    if (k < nm) {
      double sn, cs;
      sincos(double(k) * q[3], &sn, &cs);
      q[kBasisHead + 2 * k] = cs;
      q[kBasisHead + 2 * k + 1] = sn;
    } else {
      int l = 0, m = k - nm;
      while (m > l) { m -= l + 1; ++l; }
      q[kBasisHead + 2 * nm + k - nm] = sphLegendre(l, m, q[1], q[2]);
    }
  }
  __syncthreads();
  for (int t = tid; t < np * nb; t += 256) {
    int const b = t % nb;
    double const * q = sm + (t / nb) * per;
    double const * ang = q + kBasisHead;
    double const * leg = ang + 2 * nm;
    int64_t const idx = i0 * nb + t;
    DevSto const s = sto[b];
    double R, dR;
    basisRadial(s, q[0], R, dR);
    int const am = s.m < 0 ? -s.m : s.m;
    double const P = leg[s.l * (s.l + 1) / 2 + am];
    double const cs = ang[2 * am], sn = s.m < 0 ? -ang[2 * am + 1] : ang[2 * am + 1];   // of m phi
    double const rp = R * P;
    double pr;
    if (s.rtype == 0) pr = rp;
    else if (s.rtype == 1) pr = 1.4142135623730950488 * rp * cs;
    else pr = -1.4142135623730950488 * rp * sn;
    phiR[idx] = pr;
    if (vals) {
      if (ndim == 3) reinterpret_cast<double2 *>(vals)[idx] = make_double2(rp * cs, rp * sn);
      else vals[idx] = rp * cs;
    }
    if (grads) {
      // SlaterTypeOrbital.hpp:63-106 (including its m < 0 and pole behaviour), its quotients by the point's reciprocals
      double const l = s.l, m = s.m;
      double const ylmRe = P * cs, ylmIm = P * sn;
      double const c1 = (s.l != s.m) ? sqrt((l - m) * (l + m + 1)) : 0.0;
      int const m1 = s.m + 1, am1 = m1 < 0 ? -m1 : m1;
      double const P1 = am1 > s.l ? 0.0 : leg[s.l * (s.l + 1) / 2 + am1];
      double const cs1 = ang[2 * am1], sn1 = m1 < 0 ? -ang[2 * am1 + 1] : ang[2 * am1 + 1];
      double const cp = ang[2], sp = ang[3];   // of phi
      // cExp(-phi) * Y_l^{m+1}
      double const y1Re = P1 * cs1, y1Im = P1 * sn1;
      double const ylmp1Re = c1 * (cp * y1Re + sp * y1Im);
      double const ylmp1Im = c1 * (cp * y1Im - sp * y1Re);
      double const rHatRe = dR * ylmRe, rHatIm = dR * ylmIm;
      double const Rr = R * q[4], sth = q[7], cth = q[8];
      double const thRe = (m * ylmRe * q[5] + ylmp1Re) * Rr;
      double const thIm = (m * ylmIm * q[5] + ylmp1Im) * Rr;
      // i m Ylm R / (r sin t)
      double const phRe = -m * ylmIm * R * q[6];
      double const phIm = m * ylmRe * R * q[6];
      double const rx = cp * sth, ry = sp * sth, tx = cp * cth, ty = sp * cth;
      double2 * g = reinterpret_cast<double2 *>(grads) + 3 * idx;
      g[0] = make_double2(rHatRe * rx + thRe * tx - phRe * sp, rHatIm * rx + thIm * tx - phIm * sp);
      g[1] = make_double2(rHatRe * ry + thRe * ty + phRe * cp, rHatIm * ry + thIm * ty + phIm * cp);
      g[2] = make_double2(rHatRe * cth - thRe * sth, rHatIm * cth - thIm * sth);
    }
  }
}

// ---- compensated block reduction helpers -------------------------------------------------------
__device__ __forceinline__ void twoSum(double a, double b, double & s, double & e)
{
  s = a + b;
  double const bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// S_ij = sum_p w conj(v_i) v_j and, with gradients, H_ij = sum_p w (conj(g_i) . g_j / 2 - Z conj(v_i) v_j / r) over complex
// reference-basis values and gradients: a complex A^H B with two rows (S), or five (S; three gradient
// components and the value of H), per point, on the FP64 tensor cores.  A k step of 4 holds two complex
// rows, re and im apart: the real result multiplies (a.re, a.im) by (b.re, b.im), the imaginary one (a.re, -a.im) by
// (b.im, b.re), so fragments are plain 8-byte loads and the sign goes with the weight of A.  One block: a 32 x 32 tile (i tile <= j tile: S and H are Hermitian, the rest
// is mirrored) over a chunk of points, 4 warps of 8 x 32; the points' values pass through shared memory 8 at
// a time, the next ones loaded into registers meanwhile.  chunks == 1 writes S and H, else the partials
// [chunk][S, and H with gradients][nb][nb] for kQuadSum.  Bound by the FP64 MMAs.  One block per element, reading two columns with
// a stride of nb: 59,000 points x 40 functions 2,995 -> 334 us.
constexpr int kQuadPts = 8;
struct QuadArgs {
  int64_t n, chunk;
  int nb, Z;
  const double * pts;
  const double * w;
  const double2 * vals;
  const double2 * grads;   // null: S only
  double2 * S;             // [nb][nb], or the partials of chunk 0 (chunk c at S + c stride)
  double2 * H;
  int64_t stride;
};
template <bool GRAD>
__global__ void __launch_bounds__(128, 3) kQuadOverlapCore(QuadArgs a)
{
  constexpr int ROW = GRAD ? 128 : 32;   // a point's 32 values, then its 32 x 3 gradient components as stored
  constexpr int LD = ROW + 1, VPT = kQuadPts * ROW / 128;
  __shared__ double2 sA[kQuadPts][LD], sB[kQuadPts][LD];
  __shared__ double sw[kQuadPts], sz[kQuadPts];
  int const nb = a.nb, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fq = lane & 3;
  int ti = 0, tj = blockIdx.y;         // tile pair of the upper triangle, row by row
  for (int left = (nb + 31) / 32; tj >= left; --left, ++ti) tj -= left;
  tj += ti;
  int const i0 = ti * 32, j0 = tj * 32;
  int64_t const pbeg = int64_t(blockIdx.x) * a.chunk, pend = min(a.n, pbeg + a.chunk);
  double acc[GRAD ? 2 : 1][4][2][2];   // S / H, column tile, re / im, fragment element
#pragma unroll
  for (int m = 0; m < (GRAD ? 2 : 1); ++m)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[m][j][0][0] = acc[m][j][0][1] = acc[m][j][1][0] = acc[m][j][1][1] = 0.0;
  double2 av[VPT], bv[VPT];
  double wv = 0, zv = 0;
  // element e of a point's row for the tile from column c0: contiguous over the lanes in both arrays
  auto value = [&](int64_t p, int e, int c0) {
    if (e < 32) return p < pend && c0 + e < nb ? a.vals[p * nb + c0 + e] : make_double2(0, 0);
    return p < pend && 3 * c0 + e - 32 < 3 * nb ? a.grads[(p * nb + c0) * 3 + e - 32] : make_double2(0, 0);
  };
  auto load = [&](int64_t p0) {
#pragma unroll
    for (int q = 0; q < VPT; ++q) {
      int const idx = tid + 128 * q;
      av[q] = value(p0 + idx / ROW, idx % ROW, i0);
      if (i0 != j0) bv[q] = value(p0 + idx / ROW, idx % ROW, j0);
    }
    if (tid < kQuadPts) {
      int64_t const p = p0 + tid;
      bool const in = p < pend;
      wv = in ? a.w[p] : 0.0;
      zv = in && GRAD ? -a.Z * wv / norm3d(a.pts[p], a.pts[a.n + p], a.pts[2 * a.n + p]) : 0.0;
    }
  };
  load(pbeg);
  int const part = fq & 1, half = fq >> 1;   // k = 4 rows: complex row 2 s + half, re (0) or im (1)
  double2(*const sJ)[LD] = i0 != j0 ? sB : sA;
  for (int64_t p0 = pbeg; p0 < pend; p0 += kQuadPts) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < VPT; ++q) {
      int const idx = tid + 128 * q;
      sA[idx / ROW][idx % ROW] = av[q];
      if (i0 != j0) sB[idx / ROW][idx % ROW] = bv[q];
    }
    if (tid < kQuadPts) { sw[tid] = wv; sz[tid] = zv; }
    __syncthreads();
    if (p0 + kQuadPts < pend) load(p0 + kQuadPts);
    // one k step: of point p the complex row whose column c is element e0 + es c, weight f
    auto step = [&](int m, int p, int e0, int es, double f) {
      const double * x = reinterpret_cast<const double *>(&sA[p][e0 + es * (8 * warp + fr)]);
      const double * y = reinterpret_cast<const double *>(&sJ[p][e0 + es * fr]);
      double const af = f * x[part], ai = part ? -af : af;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        dmma(acc[m][j][0], af, y[16 * es * j + part]);
        dmma(acc[m][j][1], ai, y[16 * es * j + 1 - part]);
      }
    };
#pragma unroll 2
    for (int p = 0; p < kQuadPts; p += 2) step(0, p + half, 0, 1, sw[p + half]);   // S: the values of two points
    if constexpr (GRAD) {
#pragma unroll 2
      for (int p = 0; p < kQuadPts; ++p) {
        step(1, p, half ? 33 : 0, half ? 3 : 1, half ? 0.5 * sw[p] : sz[p]);   // H: value and second component,
        step(1, p, half ? 34 : 32, 3, 0.5 * sw[p]);                            // first and third
      }
    }
  }
#pragma unroll
  for (int m = 0; m < (GRAD ? 2 : 1); ++m) {
    double2 * out = (m ? a.H : a.S) + blockIdx.x * a.stride;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        int const i = i0 + 8 * warp + fr, c = j0 + 8 * j + 2 * fq + e;
        if (i >= nb || c >= nb) continue;
        double2 const v = make_double2(acc[m][j][0][e], acc[m][j][1][e]);
        out[i * nb + c] = v;
        if (ti != tj) out[c * nb + i] = make_double2(v.x, -v.y);
      }
  }
}

// S_ij and (with gradients) H_ij for small sums: one block per (i, j), the threads over the points.  Latency bound; its reads of two
// columns nb apart cost more than the tiles' MMAs only from some size on (quadPerElement)
__global__ void __launch_bounds__(256) kQuadElements(int64_t n, int nb, int Z, const double * pts, const double * w, const double2 * vals,
                                                     const double2 * grads, double2 * S, double2 * H)
{
  int const i = blockIdx.x / nb, j = blockIdx.x % nb;
  double v[4] = {0, 0, 0, 0};   // S and H, re and im
  for (int64_t p = threadIdx.x; p < n; p += blockDim.x) {
    double2 const a = vals[p * nb + i], b = vals[p * nb + j];
    double const ovRe = a.x * b.x + a.y * b.y, ovIm = a.x * b.y - a.y * b.x;   // conj(a) b
    v[0] += w[p] * ovRe;
    v[1] += w[p] * ovIm;
    if (grads) {
      double const r = norm3d(pts[p], pts[n + p], pts[2 * n + p]);
      double kRe = 0, kIm = 0;
      for (int d = 0; d < 3; ++d) {
        double2 const ga = grads[(p * nb + i) * 3 + d], gb = grads[(p * nb + j) * 3 + d];
        kRe += ga.x * gb.x + ga.y * gb.y;
        kIm += ga.x * gb.y - ga.y * gb.x;
      }
      v[2] += w[p] * (0.5 * kRe - Z * ovRe / r);
      v[3] += w[p] * (0.5 * kIm - Z * ovIm / r);
    }
  }
  __shared__ double red[8][4];
  for (int q = 0; q < 4; ++q) {
    for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][q] = v[q];
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int q = 0; q < 4; ++q)
    for (int k = 1; k < 8; ++k) v[q] += red[k][q];
  S[blockIdx.x] = make_double2(v[0], v[1]);
  if (grads) H[blockIdx.x] = make_double2(v[2], v[3]);
}
// Where one block per element is the faster form.  Its time grows with n (latency of a thread's points) and n nb^2 (reads); the tiles'
// starts higher (a second launch, 8-point groups of whole 32 x 32 tiles) and stays flat up to about 8,000 points.  Whole calls,
// per element / tiled: with H 37 / 55 us at 50 points and 47 / 59 at 2,500 (1 function), 46 / 61 at 500 and 70 / 60 at
// 2,500 (20), 74 / 65 at 500 (40); S alone 22 / 33 at 50 points, 43 / 46 at 32,768 (5), 33 / 35 at 2,500 (20), 60 / 37 (40)
bool quadPerElement(int64_t n, int nb, bool withH)
{
  return nb <= 48 && (withH ? n * (nb * nb + 100) <= 610000 : n * (nb * nb + 20) <= 1800000);
}

// out[e] = sum over the chunks c of part[c n + e]: 32 elements per block, 8 warps taking every eighth chunk each, added in warp order
__global__ void __launch_bounds__(256) kQuadSum(int n, int chunks, const double2 * part, double2 * out)
{
  __shared__ double2 red[8][32];
  int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = blockIdx.x * 32 + lane;
  double2 s = make_double2(0, 0);
  if (e < n)
#pragma unroll 4
    for (int c = warp; c < chunks; c += 8) {
      double2 const v = part[int64_t(c) * n + e];
      s.x += v.x;
      s.y += v.y;
    }
  red[warp][lane] = s;
  __syncthreads();
  if (warp != 0 || e >= n) return;
  for (int k = 1; k < 8; ++k) { s.x += red[k][lane].x; s.y += red[k][lane].y; }
  out[e] = s;
}

// S and (withH) H of a grid into out[0 .. nb^2) and out[nb^2 .. 2 nb^2); the partial sums of up to maxChunks point chunks
// go behind them (maxChunks 1: none).  Three blocks per SM (as many as are resident) where the chunks allow
constexpr int kQuadMaxChunks = 256;
int quadChunks(tcscf_ctx * ctx, Grid const & g)
{
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  int const t = (g.nb + 31) / 32, pairs = t * (t + 1) / 2;
  int64_t const want = 3 * int64_t(sms) / pairs;
  return int(std::max<int64_t>(1, std::min<int64_t>({want, kQuadMaxChunks, (g.n + 4 * kQuadPts - 1) / (4 * kQuadPts)})));
}
int quadLaunch(tcscf_ctx * ctx, Grid const & g, int Z, bool withH, double2 * out, int maxChunks)
{
  int const nb = g.nb, nn = nb * nb, t = (nb + 31) / 32;
  if (quadPerElement(g.n, nb, withH)) {
    kQuadElements<<<unsigned(nn), 256, 0, ctx->stream>>>(g.n, nb, Z, g.pts, g.w, reinterpret_cast<const double2 *>(g.vals),
                                                       withH ? reinterpret_cast<const double2 *>(g.grads) : nullptr, out, out + nn);
    TCSCF_LAUNCH(ctx);
    return TCSCF_OK;
  }
  int const want = std::min(maxChunks, quadChunks(ctx, g));
  int64_t const chunk = ((g.n + want - 1) / want + kQuadPts - 1) / kQuadPts * kQuadPts;
  int const chunks = int((g.n + chunk - 1) / chunk);
  double2 * part = chunks == 1 ? out : out + 2 * nn;
  int const m = (withH ? 2 : 1) * nn;   // elements of a chunk's partials: without H only those of S exist
  QuadArgs a{g.n, chunk, nb, Z, g.pts, g.w, reinterpret_cast<const double2 *>(g.vals), withH ? reinterpret_cast<const double2 *>(g.grads) : nullptr,
             part, part + nn, m};
  dim3 const grid{unsigned(chunks), unsigned(t * (t + 1) / 2)};
  if (withH) kQuadOverlapCore<true><<<grid, 128, 0, ctx->stream>>>(a);
  else kQuadOverlapCore<false><<<grid, 128, 0, ctx->stream>>>(a);
  TCSCF_LAUNCH(ctx);
  if (chunks > 1) {
    kQuadSum<<<unsigned((m + 31) / 32), 256, 0, ctx->stream>>>(m, chunks, part, out);
    TCSCF_LAUNCH(ctx);
  }
  return TCSCF_OK;
}

// Fixed scratch of tcscf_overlap_core_quadrature_static: S, H and the chunk partials that fit behind them (2 MiB).
constexpr int kQuadStaticMaxNb = 256;
static __device__ __align__(256) double2 gQuadStaticScratch[2 * kQuadStaticMaxNb * kQuadStaticMaxNb];

// Device address of gQuadStaticScratch on the context's device, looked up once per device with that
// device current (the caller has made it current).
int quadStaticScratch(tcscf_ctx * ctx, double2 ** out)
{
  constexpr int kMaxDevices = 64;
  static std::mutex lock;
  static double2 * addr[kMaxDevices] = {};
  TCSCF_CHECK(ctx, ctx->device >= 0 && ctx->device < kMaxDevices, TCSCF_ERR_INVALID_ARGUMENT, "device index out of range");
  std::lock_guard<std::mutex> guard(lock);
  if (!addr[ctx->device]) {
    void * p = nullptr;
    cudaError_t const e = cudaGetSymbolAddress(&p, gQuadStaticScratch);
    if (e != cudaSuccess) return fail(ctx, TCSCF_ERR_CUDA, std::string("cudaGetSymbolAddress(gQuadStaticScratch): ") + cudaGetErrorString(e));
    addr[ctx->device] = static_cast<double2 *>(p);
  }
  *out = addr[ctx->device];
  return TCSCF_OK;
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// symmetric real part (column-major == row-major) and the imaginary magnitude, per spin
__global__ void kSplitDensity(int nb, const double2 * DR, double * A, double * maxAbs)
{
  __shared__ double sre[256], sim[256];
  double mr = 0, mi = 0;
  for (int idx = threadIdx.x; idx < nb * nb; idx += blockDim.x) {
    int const k = idx / nb, l = idx % nb;
    double2 const a = DR[k * nb + l], b = DR[l * nb + k];
    A[idx] = 0.5 * (a.x + b.x);
    mr = fmax(mr, fabs(a.x));
    mi = fmax(mi, fabs(a.y));
  }
  sre[threadIdx.x] = mr;
  sim[threadIdx.x] = mi;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) { sre[threadIdx.x] = fmax(sre[threadIdx.x], sre[threadIdx.x + o]); sim[threadIdx.x] = fmax(sim[threadIdx.x], sim[threadIdx.x + o]); }
    __syncthreads();
  }
  if (threadIdx.x == 0) { maxAbs[0] = sre[0]; maxAbs[1] = sim[0]; }
}

// Hermitian (conj-symmetrised) copy of DR, column-major, for the complex factorisation
__global__ void kHermitianCopy(int nb, const double2 * DR, double2 * Z)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nb; idx += gridDim.x * blockDim.x) {
    int const row = idx % nb, col = idx / nb;   // column-major element (row, col)
    double2 const a = DR[row * nb + col], b = DR[col * nb + row];
    Z[idx] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
  }
}

constexpr int kCholeskyMaxNb = 128;

// One density factorisation (FactorBufs below): D complex [nb][nb] in the reference basis, DR its real-harmonic form,
// A the symmetrised real part, X1 and X2 the factors [nb][ldx], status {max |Re DR|, max |Im DR|, rank, indefinite}
struct FactorStatus {
  double maxAbs[2];
  int rank, indefinite;
};
struct FactorJob {
  int nb, ldx;
  const DevSto * sto;
  const double2 * D;
  double2 * DR;
  double * A, * X1, * X2;
  FactorStatus * status;
};

// element (k, l) of conj(U) D U^T
__device__ __forceinline__ double2 densityToReal(int nb, const DevSto * s, const double2 * D, int k, int l)
{
  int const ik[2] = {k, s[k].partner};
  int const jl[2] = {l, s[l].partner};
  double2 acc = make_double2(0, 0);
  for (int a = 0; a < 2; ++a) {
    int const i = ik[a];
    if (i < 0) continue;
    double2 const u1 = cconj(uRow(s, k, i));
    for (int b = 0; b < 2; ++b) {
      int const j = jl[b];
      if (j < 0) continue;
      double2 const t = cmul(cmul(u1, D[i * nb + j]), uRow(s, l, j));
      acc.x += t.x;
      acc.y += t.y;
    }
  }
  return acc;
}

// DR = conj(U) D U^T; D complex [nb][nb] (reference basis)
__global__ void kDensityToReal(int nb, const DevSto * s, const double2 * D, double2 * DR)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nb; idx += gridDim.x * blockDim.x) DR[idx] = densityToReal(nb, s, D, idx / nb, idx % nb);
}

// The whole factorisation of a density in one block of 256 threads (one block per job: a batch's densities in one
// launch), so that a single build pays one launch for what four kernels did and a batch does not run one block
// at a time.  (1) DR, A and the magnitudes.  (2) Pivoted (diagonal-pivoting) Cholesky factorisation of A:
// A = L L^T with the R columns of L written to X1 and X2; stops when the largest remaining diagonal is <=
// 1e-12 of the largest initial one; indefinite = 1 when the remainder is not negligible (largest |entry|
// above 1e-10 of the largest initial diagonal: the caller factors the density by eigen-decomposition).
// (3) One-sided Jacobi (Hestenes) orthogonalisation of L's columns (skipped when indefinite): L <- L W
// with W orthogonal; X X^T = L L^T is unchanged and X's columns become the density's eigenvectors
// scaled by the square roots of its eigenvalues (the factor the fixed-point and TF32 contractions are
// accurate with: no cancellation between columns).  Column pairs in round-robin order, one pair per warp
// at a time; at most 30 sweeps, ending when every pair is orthogonal to 1e-15 of its norms.  Bound by the
// latency of its chain of barriers (a few per pivot and Jacobi step); shared memory nb * nb doubles;
// bases above kCholeskyMaxNb take step (1) only and are marked indefinite.
__global__ void __launch_bounds__(256) kFactorDensity(FactorJob one, const FactorJob * jobs)
{
  extern __shared__ double S[];
  __shared__ double lcol[kCholeskyMaxNb];
  __shared__ int done[kCholeskyMaxNb];
  __shared__ double rv[8], rw[8];
  __shared__ int ri[8];
  __shared__ int rotated;
  FactorJob const f = jobs ? jobs[blockIdx.x] : one;
  int const nb = f.nb, ldx = f.ldx, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  double mr = 0, mi = 0;
  for (int idx = t; idx < nb * nb; idx += 256) {
    double2 const d = densityToReal(nb, f.sto, f.D, idx / nb, idx % nb);
    f.DR[idx] = d;
    mr = fmax(mr, fabs(d.x));
    mi = fmax(mi, fabs(d.y));
  }
  for (int o = 16; o > 0; o >>= 1) {
    mr = fmax(mr, __shfl_xor_sync(0xffffffffu, mr, o));
    mi = fmax(mi, __shfl_xor_sync(0xffffffffu, mi, o));
  }
  if (lane == 0) { rv[warp] = mr; rw[warp] = mi; }
  __syncthreads();   // and DR is visible to the block
  if (t == 0) {
    for (int k = 1; k < 8; ++k) { mr = fmax(mr, rv[k]); mi = fmax(mi, rw[k]); }
    f.status->maxAbs[0] = mr;
    f.status->maxAbs[1] = mi;
  }
  bool const small = nb <= kCholeskyMaxNb;
  for (int idx = t; idx < nb * nb; idx += 256) {
    int const k = idx / nb, l = idx % nb;
    double const v = 0.5 * (f.DR[idx].x + f.DR[l * nb + k].x);
    f.A[idx] = v;
    if (small) S[idx] = v;
  }
  if (!small) {
    if (t == 0) { f.status->rank = 0; f.status->indefinite = 1; }
    return;
  }
  for (int i = t; i < nb; i += 256) done[i] = 0;
  __syncthreads();
  // block reduction of (value, index): largest value, smallest index among equals
  auto better = [](double w, int wi, double v, int i) { return w > v || (w == v && wi >= 0 && (i < 0 || wi < i)); };
  auto argmax = [&](double v, int idx, double & bv, int & bi) {
    for (int o = 16; o > 0; o >>= 1) {
      double const w = __shfl_xor_sync(0xffffffffu, v, o);
      int const wi = __shfl_xor_sync(0xffffffffu, idx, o);
      if (better(w, wi, v, idx)) { v = w; idx = wi; }
    }
    if (lane == 0) { rv[warp] = v; ri[warp] = idx; }
    __syncthreads();
    bv = rv[0];
    bi = ri[0];
    for (int k = 1; k < 8; ++k)
      if (better(rv[k], ri[k], bv, bi)) { bv = rv[k]; bi = ri[k]; }
    __syncthreads();
  };
  double d0 = 0;
  int unused = 0;
  {
    double m = 0;
    for (int i = t; i < nb; i += 256) m = fmax(m, S[i * nb + i]);
    argmax(m, -1, d0, unused);
  }
  double const tol = 1e-12 * d0;
  int R = 0;
  for (; R < nb; ++R) {
    double best = -1.0;
    int bi = -1;
    for (int i = t; i < nb; i += 256)
      if (!done[i] && S[i * nb + i] > best) { best = S[i * nb + i]; bi = i; }
    double pv;
    int p;
    argmax(best, bi, pv, p);
    if (p < 0 || !(pv > tol)) break;
    double const sq = sqrt(pv), inv = 1.0 / sq;
    for (int i = t; i < nb; i += 256) {
      double const l = done[i] ? 0.0 : (i == p ? sq : S[i * nb + p] * inv);
      lcol[i] = l;
      f.X1[int64_t(i) * ldx + R] = l;
    }
    __syncthreads();
    for (int idx = t; idx < nb * nb; idx += 256) S[idx] -= lcol[idx / nb] * lcol[idx % nb];
    if (t == 0) done[p] = 1;
    __syncthreads();
  }
  double r = 0;
  for (int idx = t; idx < nb * nb; idx += 256)
    if (!done[idx / nb] && !done[idx % nb]) r = fmax(r, fabs(S[idx]));
  double rmax;
  argmax(r, -1, rmax, unused);
  bool const indefinite = rmax > 1e-10 * d0 || !(rmax == rmax);
  if (t == 0) {
    f.status->rank = R;
    f.status->indefinite = indefinite ? 1 : 0;
  }
  if (indefinite) return;
  double * Lc = S;   // [R][nb]: column a at Lc + a * nb (argmax ended with a barrier)
  for (int idx = t; idx < R * nb; idx += 256) Lc[idx] = f.X1[int64_t(idx % nb) * ldx + idx / nb];
  __syncthreads();
  int const Rp = R + (R & 1);   // an even number of slots (the last one idle when R is odd)
  for (int sweep = 0; sweep < 30 && R > 1; ++sweep) {
    if (t == 0) rotated = 0;
    __syncthreads();
    for (int step = 0; step < Rp - 1; ++step) {
      for (int k = warp; k < Rp / 2; k += 8) {
        int const a = k == 0 ? Rp - 1 : (step + k) % (Rp - 1);
        int const b = k == 0 ? step : (step - k + Rp - 1) % (Rp - 1);
        if (a >= R || b >= R) continue;
        double * ca = Lc + a * nb;
        double * cb = Lc + b * nb;
        double al = 0, be = 0, ga = 0;
        for (int i = lane; i < nb; i += 32) {
          al += ca[i] * ca[i];
          be += cb[i] * cb[i];
          ga += ca[i] * cb[i];
        }
        for (int o = 16; o > 0; o >>= 1) {
          al += __shfl_xor_sync(0xffffffffu, al, o);
          be += __shfl_xor_sync(0xffffffffu, be, o);
          ga += __shfl_xor_sync(0xffffffffu, ga, o);
        }
        if (!(fabs(ga) > 1e-15 * sqrt(al * be))) continue;
        double const zeta = (be - al) / (2.0 * ga);
        double const tn = copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        double const c = 1.0 / sqrt(1.0 + tn * tn), sn = c * tn;
        for (int i = lane; i < nb; i += 32) {
          double const x = ca[i], y = cb[i];
          ca[i] = c * x - sn * y;
          cb[i] = sn * x + c * y;
        }
        if (lane == 0) rotated = 1;
      }
      __syncthreads();
    }
    if (!rotated) break;
    __syncthreads();
  }
  for (int idx = t; idx < R * nb; idx += 256) {
    int64_t const o = int64_t(idx % nb) * ldx + idx / nb;
    f.X1[o] = Lc[idx];
    f.X2[o] = Lc[idx];
  }
}

// factor matrices X1, X2 [nb][ldx] from the kept eigenpairs (real case): X2 = v sqrt|l|, X1 = sign(l) X2
__global__ void kRealFactors(int nb, int nkeep, const int * keep, const double * W, const double * V, int ldx, double * X1, double * X2)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nkeep; idx += gridDim.x * blockDim.x) {
    int const k = idx / nkeep, b = idx % nkeep;
    int const e = keep[b];
    double const lam = W[e];
    double const sq = sqrt(fabs(lam));
    double const v = V[e * nb + k] * sq;
    X2[k * ldx + b] = v;
    X1[k * ldx + b] = lam < 0 ? -v : v;
  }
}

// complex case: X2 = [Re z | Im z], X1re = [l Re z | l Im z], X1im = [l Im z | -l Re z]
__global__ void kComplexFactors(int nb, int nkeep, const int * keep, const double * W, const double2 * Z, int ldx, double * X1re,
                                double * X1im, double * X2)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nkeep; idx += gridDim.x * blockDim.x) {
    int const k = idx / nkeep, b = idx % nkeep;
    int const e = keep[b];
    double const lam = W[e];
    double2 const z = Z[e * nb + k];
    X2[k * ldx + b] = z.x;
    X2[k * ldx + nkeep + b] = z.y;
    X1re[k * ldx + b] = lam * z.x;
    X1re[k * ldx + nkeep + b] = lam * z.y;
    X1im[k * ldx + b] = lam * z.y;
    X1im[k * ldx + nkeep + b] = -lam * z.x;
  }
}

// One side of a contraction from one read of the basis values phi [n][nb]: psi[r][b] = sum_k phi[r][k] X[k][b] for
// b < R (row stride ld); with coul, coul[r] = scale w[r] sum_b psi'[r][b] psi[r][b], psi' from the factor Xc (null: psi
// itself); with V, V[r][l] = scale w[r] phi[r][l].  A block takes `rows` points (8 per warp): phi rows and the factors in
// shared memory (rows 4 mod 16 doubles apart: conflict-free fragments), the products on the FP64 tensor
// cores, four column tiles at a time.  Bound by HBM.  As three kernels, each reading its operands again (one
// thread per (r, b), the phi row from global memory): Kr (406,000 points, 120 columns, rank 18) 984 -> 375 us.
// The functions pass through shared memory `panel` (a multiple of 4) at a time: all of them where they fit, and bases of about a
// thousand functions and more in panels that are read again for every 32 columns
struct OrbitalArgs {
  int64_t n;
  int nb, R, ldx, ld, rows, panel;
  double scale;
  const double * phi;
  const double * w;
  const double * X;
  const double * Xc;
  double * psi;
  double * coul;
  double * V;
};
__global__ void __launch_bounds__(256) kOrbitals(OrbitalArgs a)
{
  extern __shared__ double sm[];
  int const nb = a.nb, nb4 = (nb + 3) / 4 * 4, kp = a.panel, R8 = (a.R + 7) / 8 * 8, lp = fragStride(kp), lx = fragStride(R8);
  int const t = threadIdx.x, warp = t >> 5, lane = t & 31, fr = lane >> 2, fq = lane & 3;
  double * sX = sm;                                // [kp][lx], then the same of Xc
  double * sXc = sX + kp * lx;
  double * sPhi = sXc + (a.Xc ? kp * lx : 0);      // [rows][lp]
  int64_t const r0 = int64_t(blockIdx.x) * a.rows;
  int const nr = int(min(int64_t(a.rows), a.n - r0));
  auto load = [&](int k0, int kn) {
    for (int k = warp; k < kn; k += 8)
      for (int b = lane; b < R8; b += 32) {
        bool const in = k0 + k < nb && b < a.R;
        sX[k * lx + b] = in ? a.X[int64_t(k0 + k) * a.ldx + b] : 0.0;
        if (a.Xc) sXc[k * lx + b] = in ? a.Xc[int64_t(k0 + k) * a.ldx + b] : 0.0;
      }
    // with all functions in one panel the block's phi rows are one contiguous range: every load in flight at once
    for (int r = warp; r < a.rows; r += 8)
#pragma unroll 4
      for (int c = lane; c < kn; c += 32) {
        bool const in = r < nr && k0 + c < nb;
        cpAsync<8>(&sPhi[r * lp + c], in ? a.phi + (r0 + r) * nb + k0 + c : a.phi, in ? 8 : 0);
      }
    cpAsyncCommit();
    cpAsyncWait<0>();
    __syncthreads();
  };
  int const row = 8 * warp + fr;
  double s = 0;
  for (int b0 = 0; b0 < R8; b0 += 32) {
    double q[4][2], qc[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j][0] = q[j][1] = qc[j][0] = qc[j][1] = 0.0;
    for (int k0 = 0; k0 < nb4; k0 += kp) {
      int const kn = min(kp, nb4 - k0);
      if (b0 == 0 || kp < nb4) {
        if (b0 + k0 > 0) __syncthreads();   // every warp is done with the panel before
        load(k0, kn);
        if (a.V && b0 == 0)
          for (int r = warp; r < nr; r += 8) {
            double const f = a.scale * a.w[r0 + r];
#pragma unroll 4
            for (int c = lane; c < min(kn, nb - k0); c += 32) a.V[(r0 + r) * nb + k0 + c] = f * sPhi[r * lp + c];
          }
      }
      if (8 * warp >= a.rows) continue;
      for (int k = fq; k < kn; k += 4) {
        double const p = sPhi[row * lp + k];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (b0 + 8 * j < R8) dmma(q[j], p, sX[k * lx + b0 + 8 * j + fr]);
        if (a.Xc) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (b0 + 8 * j < R8) dmma(qc[j], p, sXc[k * lx + b0 + 8 * j + fr]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        int const b = b0 + 8 * j + 2 * fq + e;
        if (row < nr && b < a.R) a.psi[(r0 + row) * a.ld + b] = q[j][e];
        s = fma(a.Xc ? qc[j][e] : q[j][e], q[j][e], s);   // columns past R are zero
      }
  }
  if (!a.coul) return;
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  if (fq == 0 && row < nr) a.coul[r0 + row] = a.scale * a.w[r0 + row] * s;
}

int orbitals(tcscf_ctx * ctx, OrbitalArgs a)
{
  // the limit of the entry points, and its status, as they have always been
  TCSCF_CHECK(ctx, size_t(a.nb) * a.R * sizeof(double) <= 48 * 1024, TCSCF_ERR_CUDA, "orbital factor (basis size x density rank) above 6144 elements");
  int const R8 = (a.R + 7) / 8 * 8;
  auto bytes = [&](int rows) { return sizeof(double) * (size_t(a.panel) * fragStride(R8) * (a.Xc ? 2 : 1) + size_t(rows) * fragStride(a.panel)); };
  a.panel = (a.nb + 3) / 4 * 4;
  a.rows = 64;
  while (a.rows > 8 && bytes(a.rows) > 200 * 1024) a.rows /= 2;
  if (bytes(a.rows) > 227 * 1024) { a.panel = 256; a.rows = 64; }   // more than 908 functions, so at most 6 columns: 182 KB
  TCSCF_CHECK(ctx, bytes(a.rows) <= 227 * 1024, TCSCF_ERR_UNSUPPORTED, "internal: orbital panel beyond the shared memory");
  TCSCF_CUDA(ctx, cudaFuncSetAttribute(kOrbitals, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes(a.rows))));
  kOrbitals<<<unsigned((a.n + a.rows - 1) / a.rows), 256, bytes(a.rows), ctx->stream>>>(a);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

// V[r][l] = scale w[r] phi[r][l] (kOrbitals writes it beside a factor's orbitals)
__global__ void kWeightedBasis(int64_t n, int nb, const double * phi, const double * w, double scale, double * V)
{
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < n * nb; idx += int64_t(gridDim.x) * blockDim.x)
    V[idx] = scale * w[idx / nb] * phi[idx];
}

// V[r][p(k,l)] = scale w[r] phi[r][k] phi[r][l], k <= l, pair index p = k*nb - k(k-1)/2 + (l-k)
__global__ void kPairProducts(int64_t n, int nb, const double * phi, const double * w, double scale, double * V)
{
  int const np = nb * (nb + 1) / 2;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < n * np; idx += int64_t(gridDim.x) * blockDim.x) {
    int64_t const r = idx / np;
    int p = int(idx % np);
    int k = 0;
    while (p >= nb - k) { p -= nb - k; ++k; }
    int const l = k + p;
    V[idx] = scale * w[r] * phi[r * nb + k] * phi[r * nb + l];
  }
}

__device__ __forceinline__ int pairIndex(int nb, int k, int l)
{
  if (k > l) { int t = k; k = l; l = t; }
  return k * nb - k * (k - 1) / 2 + (l - k);
}

// plane `comp` of a kept tensor (Tensor): the symmetric nb x nb matrices of the packed pair sums FR [n1][np]
__global__ void kPairsToPlanes(int64_t n1, int nb, const double * FR, int ncomp, int comp, double * out)
{
  int const np = nb * (nb + 1) / 2, ps = tensorPlane(nb), ld = tensorStride(nb);
  int64_t const total = n1 * ps;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total; idx += int64_t(gridDim.x) * blockDim.x) {
    int64_t const r = idx / ps;
    int const e = int(idx % ps);
    int const k = e / ld, l = e % ld;
    out[(r * ncomp + comp) * ps + e] = k < nb && l < nb ? FR[r * np + pairIndex(nb, k, l)] : 0.0;
  }
}

// F(j,i) = sum_{k,l} U[k][j] FR(k,l) conj(U[l][i]) for `rows` points of a kept tensor's planes: out complex [rows][nb][nb][ncomp],
// or real [rows][nb][nb] when realOut
__global__ void kPlanesToReference(int64_t rows, int nb, const DevSto * s, const double * FR, int ncomp, int realOut, double * out)
{
  int const ps = tensorPlane(nb), ld = tensorStride(nb);
  int64_t const total = rows * nb * nb * ncomp;
  for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total; idx += int64_t(gridDim.x) * blockDim.x) {
    int const comp = int(idx % ncomp);
    int64_t const e = idx / ncomp, r = e / (nb * nb);
    int const j = int((e / nb) % nb), i = int(e % nb);
    double const * F = FR + (r * ncomp + comp) * ps;
    int const kj[2] = {j, s[j].partner};
    int const li[2] = {i, s[i].partner};
    double2 acc = make_double2(0, 0);
    for (int a = 0; a < 2; ++a) {
      int const k = kj[a];
      if (k < 0) continue;
      double2 const uk = uRow(s, k, j);
      for (int b = 0; b < 2; ++b) {
        int const l = li[b];
        if (l < 0) continue;
        double const f = F[k * ld + l];
        double2 const t = cmul(uk, cconj(uRow(s, l, i)));
        acc.x += f * t.x;
        acc.y += f * t.y;
      }
    }
    if (realOut) out[idx] = acc.x;
    else reinterpret_cast<double2 *>(out)[idx] = acc;
  }
}

// element (j, i) of U^T GR conj(U) for one spin's GR (re / im planes, im may be null), GR + tr^T in its place where tr is given
__device__ __forceinline__ double2 realToReference(int nb, const DevSto * s, const double * re, const double * im, const double * tr, int j, int i)
{
  int const kj[2] = {j, s[j].partner};
  int const li[2] = {i, s[i].partner};
  double2 acc = make_double2(0, 0);
  for (int a = 0; a < 2; ++a) {
    int const k = kj[a];
    if (k < 0) continue;
    double2 const uk = uRow(s, k, j);
    for (int b = 0; b < 2; ++b) {
      int const l = li[b];
      if (l < 0) continue;
      double2 g = make_double2(re[k * nb + l], im ? im[k * nb + l] : 0.0);
      if (tr) g.x += tr[l * nb + k];
      double2 const t = cmul(cmul(uk, g), cconj(uRow(s, l, i)));
      acc.x += t.x;
      acc.y += t.y;
    }
  }
  return acc;
}
// G(j,i) = sum_{k,l} U[k][j] GR(k,l) conj(U[l][i]); GR [nspin][nb][nb] given as re/im planes
__global__ void kRealToReference(int nspin, int nb, const DevSto * s, const double * GRre, const double * GRim, double2 * G)
{
  int const nn = nb * nb;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nspin * nn; idx += gridDim.x * blockDim.x) {
    int const sp = idx / nn, ji = idx % nn;
    G[idx] = realToReference(nb, s, GRre + sp * nn, GRim ? GRim + sp * nn : nullptr, nullptr, ji / nb, ji % nb);
  }
}

// The end of a Fock build: G from the real-harmonic sums (gr.re; symSpin bit s: G = M + M^T there, or M + tr^T) or as given (gr.re null),
// enforceOneElectronSymmetry (HartreeFock.cpp:758-780), constructSCFOperator (:48-98) and the
// compensated FP64 energy, factor * Re sum D(i,j) (h(j,i) + G(j,i)/2 - G3(j,i)/3): every thread sums its terms with
// TwoSum, warps and blocks are combined in a fixed order.  parts[block] = {sum, compensation}; one block
// alone writes the energy, several leave it to kEnergySum
struct RealSums {
  const double * re;
  const double * im;
  const DevSto * sto;
  int symSpin;
  const double * tr = nullptr;
};
__device__ __forceinline__ void addPair(double & s, double & c, double s2, double c2)
{
  double t, err;
  twoSum(s, s2, t, err);
  s = t;
  c += err + c2;
}
constexpr int kFinishThreads = 256;
__global__ void __launch_bounds__(kFinishThreads) kFockFinish(int nspin, int nb, RealSums gr, const double * h, double2 * G, const double2 * G3,
                                                            const double2 * D, int respectSym, double factor, double2 * fock, double2 * parts,
                                                            double * energy)
{
  __shared__ double2 red[kFinishThreads / 32];
  double s = 0, c = 0;
  int const nn = nb * nb;
  for (int idx = blockIdx.x * kFinishThreads + threadIdx.x; idx < nspin * nn; idx += gridDim.x * kFinishThreads) {
    int const sp = idx / nn, ji = idx % nn, j = ji / nb, i = ji % nb;
    double2 g = gr.re ? realToReference(nb, gr.sto, gr.re + sp * nn, gr.im ? gr.im + sp * nn : nullptr,
                                             (gr.symSpin >> sp) & 1 ? (gr.tr ? gr.tr : gr.re) + sp * nn : nullptr, j, i) : G[idx];
    double2 g3 = G3 ? G3[idx] : make_double2(0, 0);
    if (respectSym && !(fabs(h[ji]) > 0)) { g = make_double2(0, 0); g3 = make_double2(0, 0); }
    G[idx] = g;
    double2 f = make_double2(h[ji] + g.x - g3.x, g.y - g3.y);
    if (fock) fock[idx] = f;
    double2 const e = make_double2(h[ji] + g.x / 2 - g3.x / 3, g.y / 2 - g3.y / 3);
    double2 const d = D[int64_t(sp) * nn + i * nb + j];
    addPair(s, c, d.x * e.x - d.y * e.y, 0.0);
  }
  for (int o = 16; o > 0; o >>= 1) addPair(s, c, __shfl_down_sync(0xffffffffu, s, o), __shfl_down_sync(0xffffffffu, c, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = make_double2(s, c);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kFinishThreads / 32; ++k) addPair(s, c, red[k].x, red[k].y);
    if (gridDim.x == 1) energy[0] = factor * (s + c);
    else parts[blockIdx.x] = make_double2(s, c);
  }
}
__global__ void kEnergySum(int n, const double2 * parts, double factor, double * energy)
{
  double s = 0, c = 0;
  for (int k = threadIdx.x; k < n; k += 32) addPair(s, c, parts[k].x, parts[k].y);
  for (int o = 16; o > 0; o >>= 1) addPair(s, c, __shfl_down_sync(0xffffffffu, s, o), __shfl_down_sync(0xffffffffu, c, o));
  if (threadIdx.x == 0) energy[0] = factor * (s + c);
}
int fockFinish(tcscf_ctx * ctx, int nspin, int nb, RealSums const & gr, const double * h, double2 * G, const double2 * G3, const double2 * D,
               int respectSym, double factor, double2 * fock, double * energy)
{
  // one block up to four elements a thread (a second launch costs more than they do), else up to 64
  int const n = nspin * nb * nb, blocks = n <= 4 * kFinishThreads ? 1 : std::min(64, (n + kFinishThreads - 1) / kFinishThreads);
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "fock_finish", sizeof(double2) * 64, &p));
  double2 * parts = static_cast<double2 *>(p);
  kFockFinish<<<blocks, kFinishThreads, 0, ctx->stream>>>(nspin, nb, gr, h, G, G3, D, respectSym, factor, fock, parts, energy);
  TCSCF_LAUNCH(ctx);
  if (blocks > 1) {
    kEnergySum<<<1, 32, 0, ctx->stream>>>(blocks, parts, factor, energy);
    TCSCF_LAUNCH(ctx);
  }
  return TCSCF_OK;
}

// Faa(r) = sum_ji F(r,j,i) D(i,j) (summed over the spins) and Fai_s(r,i) = sum_j (sum_k D_s(k,j) phi(r,k)) F(r,j,i)
// (calculateIaa / calculateFai, HartreeFock.cpp:144-213) in the real-harmonic basis, from a kept tensor's real
// planes, for complex D = DR [nspin][nb][nb]; re and im parts apart.  One block of 8 warps per point at a time: warp w
// takes plane rows k = w, w + 8, ... with the lanes over the columns; from the row of D^T it forms q_k = sum_m
// D(m,k) phi_m (lanes, then shuffles), the row's share of Faa, and adds q_k F(k, .) to the lanes' columns of Fai; the warps'
// sums meet in shared memory.  Every plane is read once for both spins.  The row stride and plane come as arguments (ld, ps): formed
// from nb in the kernel they cost 293 us a build where this takes 272.  Bound by HBM and the shuffles; the
// complex layout, read once per spin and sum: 16,384 points x 40 functions 337 -> 136 us, and the complex
// reduction after it (16 blocks of 1,024 rows) 1,188 -> 22 us as two real ones.
constexpr int kFaiMaxNb = 64;
template <int NSPIN>
__global__ void __launch_bounds__(256) kFaaFai(int64_t n1, int nb, int ld, int ps, const double * __restrict__ F, const double * __restrict__ phi, const double2 * DR,
                                              double * FaaRe, double * FaaIm, double * FaiRe, double * FaiIm)
{
  extern __shared__ double2 sDT[];   // [NSPIN][nb][nb]: D_s(m, k) at [s][k][m]
  __shared__ double2 sFai[8][NSPIN][kFaiMaxNb];
  __shared__ double2 sFaa[8];
  int const nn = nb * nb, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int e = tid; e < NSPIN * nn; e += 256) {
    int const s = e / nn, k = e % nn / nb, m = e % nb;
    sDT[e] = DR[s * nn + m * nb + k];
  }
  __syncthreads();
  bool const in0 = lane < nb, in1 = lane + 32 < nb;
  for (int64_t r = blockIdx.x; r < n1; r += gridDim.x) {
    double const p0 = in0 ? phi[r * nb + lane] : 0.0, p1 = in1 ? phi[r * nb + lane + 32] : 0.0;
    const double * Fr = F + r * ps;
    double2 fai[NSPIN][2], faa = make_double2(0, 0);
#pragma unroll
    for (int s = 0; s < NSPIN; ++s) fai[s][0] = fai[s][1] = make_double2(0, 0);
#pragma unroll 4
    for (int k = warp; k < nb; k += 8) {
      double const f0 = in0 ? Fr[k * ld + lane] : 0.0, f1 = in1 ? Fr[k * ld + lane + 32] : 0.0;
#pragma unroll
      for (int s = 0; s < NSPIN; ++s) {
        double2 const d0 = in0 ? sDT[s * nn + k * nb + lane] : make_double2(0, 0), d1 = in1 ? sDT[s * nn + k * nb + lane + 32] : make_double2(0, 0);
        faa.x = fma(f0, d0.x, fma(f1, d1.x, faa.x));
        faa.y = fma(f0, d0.y, fma(f1, d1.y, faa.y));
        double2 q = make_double2(fma(p0, d0.x, p1 * d1.x), fma(p0, d0.y, p1 * d1.y));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          q.x += __shfl_xor_sync(0xffffffffu, q.x, o);
          q.y += __shfl_xor_sync(0xffffffffu, q.y, o);
        }
        fai[s][0].x = fma(q.x, f0, fai[s][0].x);
        fai[s][0].y = fma(q.y, f0, fai[s][0].y);
        fai[s][1].x = fma(q.x, f1, fai[s][1].x);
        fai[s][1].y = fma(q.y, f1, fai[s][1].y);
      }
    }
#pragma unroll
    for (int s = 0; s < NSPIN; ++s) {
      if (in0) sFai[warp][s][lane] = fai[s][0];
      if (in1) sFai[warp][s][lane + 32] = fai[s][1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      faa.x += __shfl_xor_sync(0xffffffffu, faa.x, o);
      faa.y += __shfl_xor_sync(0xffffffffu, faa.y, o);
    }
    if (lane == 0) sFaa[warp] = faa;
    __syncthreads();
    for (int e = tid; e < NSPIN * nb; e += 256) {
      int const s = e / nb, i = e % nb;
      double2 a = make_double2(0, 0);
#pragma unroll
      for (int w = 0; w < 8; ++w) { a.x += sFai[w][s][i].x; a.y += sFai[w][s][i].y; }
      int64_t const o = (s * n1 + r) * nb + i;
      FaiRe[o] = a.x;
      FaiIm[o] = a.y;
    }
    if (tid == 255) {
      double2 a = make_double2(0, 0);
      for (int w = 0; w < 8; ++w) { a.x += sFaa[w].x; a.y += sFaa[w].y; }
      FaaRe[r] = a.x;
      FaaIm[r] = a.y;
    }
    __syncthreads();
  }
}

// the Coulomb potential of both spins
__global__ void kAddSpins(int64_t n, const double * a, const double * b, double * out)
{
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) out[i] = a[i] + b[i];
}

// column-major complex copy of the row-major (j,i) Fock matrix, and of a real row-major S
__global__ void kToColumnMajor(int nb, const double2 * fockRow, const double * S, double2 * A, double2 * B)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nb; idx += gridDim.x * blockDim.x) {
    int const row = idx % nb, col = idx / nb;
    A[idx] = fockRow[row * nb + col];
    B[idx] = make_double2(S[row * nb + col], 0.0);
  }
}

// getNewDensity (HartreeFock.cpp:20-44): D(u,v) = sum_a C(u,a) conj(C(v,a)); C column-major
__global__ void kDensityFromOrbitals(int nb, int nocc, const double2 * C, double2 * D)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nb; idx += gridDim.x * blockDim.x) {
    int const u = idx / nb, v = idx % nb;
    double2 t = make_double2(0, 0);
    for (int a = 0; a < nocc; ++a) {
      double2 const x = cmul(C[a * nb + u], cconj(C[a * nb + v]));
      t.x += x.x; t.y += x.y;
    }
    D[idx] = t;
  }
}

// real-harmonic density DR(u,v) = sum_a C(u,a) C(v,a) from real eigenvectors C (column-major)
__global__ void kRealDensity(int nb, int nocc, const double * C, double * DR)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nb; idx += gridDim.x * blockDim.x) {
    int const u = idx / nb, v = idx % nb;
    double t = 0;
    for (int a = 0; a < nocc; ++a) t += C[a * nb + u] * C[a * nb + v];
    DR[idx] = t;
  }
}

// the occupied eigenvectors of a real-harmonic eigen-solve (columns of the column-major C) as the
// density factor X [nb][ldx] (X[k][a] = C[a][k]): D_R = X X^T, the density kRealDensity forms
__global__ void kFactorFromOrbitals(int nb, int nocc, const double * C, int ldx, double * X)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < nb * nocc; idx += gridDim.x * blockDim.x) {
    int const k = idx / nocc, a = idx % nocc;
    X[int64_t(k) * ldx + a] = C[a * nb + k];
  }
}

// ---- Pulay DIIS (optional SCF acceleration; the reference iterates plain Roothaan steps) ---------
// dots[j] = Re <E[slot], E[j]> (Frobenius product of the commutator error matrices of both spins)
// for the used history slots j < count, one block per j
__global__ void kDiisDots(int64_t len, int slot, int count, const double2 * E, double * dots)
{
  __shared__ double red[256];
  int const j = blockIdx.x;
  if (j >= count) return;
  double acc = 0;
  for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
    double2 const a = E[int64_t(slot) * len + i], b = E[int64_t(j) * len + i];
    acc += a.x * b.x + a.y * b.y;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) dots[j] = red[0];
}

// F = sum_j c[j] Fh[j]
__global__ void kDiisCombine(int64_t len, int count, const double * c, const double2 * Fh, double2 * F)
{
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < len; i += int64_t(gridDim.x) * blockDim.x) {
    double2 a = make_double2(0, 0);
    for (int j = 0; j < count; ++j) {
      double2 const f = Fh[int64_t(j) * len + i];
      a.x += c[j] * f.x;
      a.y += c[j] * f.y;
    }
    F[i] = a;
  }
}

__global__ void kRealToComplex(int64_t n, const double * a, double2 * b)
{
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) b[i] = make_double2(a[i], 0.0);
}

// row-major C = alpha A B + beta C (n x n complex) through column-major cuBLAS: C^T = B^T A^T
int rowMajorZgemm(tcscf_ctx * ctx, cublasHandle_t h, int n, double2 alpha, const double2 * A, const double2 * B, double2 beta, double2 * C)
{
  cuDoubleComplex const al = make_cuDoubleComplex(alpha.x, alpha.y), be = make_cuDoubleComplex(beta.x, beta.y);
  if (cublasZgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, n, n, n, &al, reinterpret_cast<const cuDoubleComplex *>(B), n,
                  reinterpret_cast<const cuDoubleComplex *>(A), n, &be, reinterpret_cast<cuDoubleComplex *>(C), n) != CUBLAS_STATUS_SUCCESS)
    return fail(ctx, TCSCF_ERR_CUDA, "cublasZgemm failed");
  return TCSCF_OK;
}

// Solves the DIIS equations [B -1; -1 0] [c; lambda] = [0; -1] (B m x m, row stride ld) by Gaussian
// elimination with partial pivoting; false when singular
bool solveDiis(int m, std::vector<double> const & B, int ld, std::vector<double> & c)
{
  int const n = m + 1;
  std::vector<double> A(size_t(n) * (n + 1), 0.0);
  for (int i = 0; i < m; ++i) {
    for (int j = 0; j < m; ++j) A[i * (n + 1) + j] = B[i * ld + j];
    A[i * (n + 1) + m] = -1;
    A[m * (n + 1) + i] = -1;
  }
  A[m * (n + 1) + n] = -1;
  for (int k = 0; k < n; ++k) {
    int p = k;
    for (int i = k + 1; i < n; ++i)
      if (std::fabs(A[i * (n + 1) + k]) > std::fabs(A[p * (n + 1) + k])) p = i;
    if (!(std::fabs(A[p * (n + 1) + k]) > 0)) return false;
    if (p != k)
      for (int j = 0; j <= n; ++j) std::swap(A[k * (n + 1) + j], A[p * (n + 1) + j]);
    for (int i = k + 1; i < n; ++i) {
      double const f = A[i * (n + 1) + k] / A[k * (n + 1) + k];
      for (int j = k; j <= n; ++j) A[i * (n + 1) + j] -= f * A[k * (n + 1) + j];
    }
  }
  std::vector<double> x(n);
  for (int i = n - 1; i >= 0; --i) {
    double t = A[i * (n + 1) + n];
    for (int j = i + 1; j < n; ++j) t -= A[i * (n + 1) + j] * x[j];
    x[i] = t / A[i * (n + 1) + i];
  }
  c.assign(x.begin(), x.begin() + m);
  for (double v : c)
    if (!(v == v)) return false;
  return true;
}

}  // namespace

int finalizeLaunch(tcscf_ctx * ctx, int nspin, int nb, const double * h, double2 * G, const double2 * G3, const double2 * D, int respectSym,
                   double factor, double2 * fock, double * energy)
{
  return fockFinish(ctx, nspin, nb, RealSums{}, h, G, G3, D, respectSym, factor, fock, energy);
}

int densityToRealLaunch(tcscf_ctx * ctx, int nb, const DevSto * sto, const double2 * D, double2 * DR)
{
  kDensityToReal<<<gridBlocks(int64_t(nb) * nb, 256), 256, 0, ctx->stream>>>(nb, sto, D, DR);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

int tensorToReference(tcscf_ctx * ctx, Tensor const & t, const DevSto * sto, int64_t r0, int64_t rows, double * out)
{
  int const ncomp = t.vec ? 3 : 1;
  kPlanesToReference<<<gridBlocks(rows * t.nb * t.nb * ncomp, 256), 256, 0, ctx->stream>>>(rows, t.nb, sto, t.d + r0 * ncomp * tensorPlane(t.nb), ncomp,
                                                                                           t.isComplex ? 0 : 1, out);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

// Tensor memory comes from the context's pool: a precompute per geometry or per Jastrow trial frees and takes the same sizes
// again, which cudaMalloc and cudaFree of gigabytes made cost milliseconds to hundreds of milliseconds a call.
// A request that the pool cannot grow to is tried once more with the pool's cached memory given back
int tensorAlloc(tcscf_ctx * ctx, Tensor & t, size_t bytes)
{
  void * p = nullptr;
  if (gridAllocBytes(ctx, &p, bytes) != TCSCF_OK) {
    cudaGetLastError();
    cudaStreamSynchronize(ctx->stream);
    cudaMemPoolTrimTo(ctx->gridPool, 0);
    TCSCF_TRY(gridAllocBytes(ctx, &p, bytes));
  }
  t.d = static_cast<double *>(p);
  return TCSCF_OK;
}
void tensorRelease(tcscf_ctx * ctx, Tensor & t)
{
  gridRelease(ctx, t.d);
  t.d = nullptr;
}

// ------------------------------------------------------------------------------------------------
// Fock-build pipeline
// ------------------------------------------------------------------------------------------------
namespace {

struct Factor {
  int R = 0;          // columns of the factor matrices
  bool complex = false;
  bool same = false;  // X1 == X2 (the pivoted Cholesky factor of a positive semi-definite real density)
  double * X1 = nullptr, * X1im = nullptr, * X2 = nullptr;   // device [nb][ldx]
  int ldx = 0;
};

// Factor the spin density's real-harmonic form DR = X1 X2^T (real) or, for a density that is not
// real in the real-harmonic basis, into the real/imaginary pair described in kComplexFactors.
// Device buffers of one density factorisation: the real-harmonic density DR, its symmetrised real
// part A, the factors X1 (X1im) and X2 [nb][ldx], and the status {max |Re DR|, max |Im DR|} with the
// pivoted-Cholesky rank and flag behind it (FactorStatus).
struct FactorBufs {
  double2 * DR = nullptr;
  double * A = nullptr;
  double * X1 = nullptr, * X1im = nullptr, * X2 = nullptr;
  FactorStatus * status = nullptr;
};
size_t factorBufBytes(int nb)
{
  size_t const nn = size_t(nb) * nb;
  return nn * sizeof(double2) + nn * sizeof(double) + 3 * nn * 2 * sizeof(double) + 2 * sizeof(FactorStatus) + 256;
}
FactorBufs carveFactorBufs(void * p, int nb)
{
  size_t const nn = size_t(nb) * nb;
  char * base = static_cast<char *>(p);
  FactorBufs b;
  b.DR = reinterpret_cast<double2 *>(base); base += nn * sizeof(double2);
  b.A = reinterpret_cast<double *>(base); base += nn * sizeof(double);
  b.X1 = reinterpret_cast<double *>(base); base += nn * 2 * sizeof(double);
  b.X1im = reinterpret_cast<double *>(base); base += nn * 2 * sizeof(double);
  b.X2 = reinterpret_cast<double *>(base); base += nn * 2 * sizeof(double);
  b.status = reinterpret_cast<FactorStatus *>(base);
  return b;
}

FactorJob factorJob(Grid const & g, const double2 * dD, FactorBufs const & b)
{
  return {g.nb, 2 * g.nb, g.dsto, dD, b.DR, b.A, b.X1, b.X2, b.status};
}
// Launches (no host synchronisation) the factorisations: `one`, or the `count` jobs of a device array; maxNb: their largest basis
int factorLaunch(tcscf_ctx * ctx, FactorJob const & one, const FactorJob * jobs, int count, int maxNb)
{
  TCSCF_CUDA(ctx, cudaFuncSetAttribute(kFactorDensity, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(double) * kCholeskyMaxNb * kCholeskyMaxNb)));
  int const nb = std::min(maxNb, kCholeskyMaxNb);
  kFactorDensity<<<count, 256, sizeof(double) * nb * nb, ctx->stream>>>(one, jobs);
  TCSCF_LAUNCH(ctx);
  return TCSCF_OK;
}

// Completes the factorisation from the status read back to the host: the pivoted Cholesky factor
// with orthogonalised columns (X1 = X2 = L W) when the density is real and positive semi-definite in
// the real-harmonic basis,
// otherwise the eigen-decomposition (real: DR = X1 X2^T with X1 = V sign(l) sqrt|l|, X2 = V sqrt|l|;
// complex: the real/imaginary pair described in kComplexFactors), keeping the eigenvalues above
// 1e-12 of the largest.
int factorFinish(tcscf_ctx * ctx, Grid & g, FactorBufs const & b, FactorStatus const & st, Factor & f)
{
  int const nb = g.nb;
  size_t const nn = size_t(nb) * nb;
  f.X1 = b.X1; f.X1im = b.X1im; f.X2 = b.X2;
  f.ldx = 2 * nb;
  double const hmax[2] = {st.maxAbs[0], st.maxAbs[1]};
  if (!(hmax[0] == hmax[0]) || !(hmax[1] == hmax[1])) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite density");
  // an imaginary part below 1e-10 of the real part is rounding (SCF densities from the complex
  // eigen-solver carry ~1e-12): the density is factored as real, dropping it
  f.complex = hmax[1] > 1e-10 * std::max(hmax[0], 1e-300);
  if (hmax[0] == 0 && hmax[1] == 0) { f.R = 0; return TCSCF_OK; }
  if (!f.complex && !st.indefinite) { f.R = st.rank; f.same = true; return TCSCF_OK; }

  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "fac_eig", nn * sizeof(double2) * 2 + nn * sizeof(double) + 64 * sizeof(double) + nb * sizeof(int) + 1024, &p));
  char * base = static_cast<char *>(p);
  double2 * Z = reinterpret_cast<double2 *>(base); base += nn * sizeof(double2) * 2;
  double * W = reinterpret_cast<double *>(base); base += nn * sizeof(double);
  int * devInfo = reinterpret_cast<int *>(base); base += 64 * sizeof(double);
  int * keep = reinterpret_cast<int *>(base);
  double * A = b.A;
  int lwork = 0;
  std::vector<double> hW(nb);
  if (!f.complex) {
    if (cusolverDnDsyevd_bufferSize(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, nb, A, nb, W, &lwork) != CUSOLVER_STATUS_SUCCESS)
      return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnDsyevd_bufferSize failed");
    void * wk = nullptr;
    TCSCF_TRY(scratch(ctx, "syevd_work", size_t(lwork) * sizeof(double) + 64, &wk));
    if (cusolverDnDsyevd(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, nb, A, nb, W, static_cast<double *>(wk), lwork, devInfo) != CUSOLVER_STATUS_SUCCESS)
      return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnDsyevd failed");
  } else {
    kHermitianCopy<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, b.DR, Z);
    TCSCF_LAUNCH(ctx);
    if (cusolverDnZheevd_bufferSize(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, nb, reinterpret_cast<cuDoubleComplex *>(Z), nb, W, &lwork) != CUSOLVER_STATUS_SUCCESS)
      return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnZheevd_bufferSize failed");
    void * wk = nullptr;
    TCSCF_TRY(scratch(ctx, "heevd_work", size_t(lwork) * sizeof(double2) + 64, &wk));
    if (cusolverDnZheevd(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, nb, reinterpret_cast<cuDoubleComplex *>(Z), nb, W,
                         static_cast<cuDoubleComplex *>(wk), lwork, devInfo) != CUSOLVER_STATUS_SUCCESS)
      return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnZheevd failed");
  }
  int info = 0;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(hW.data(), W, nb * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(&info, devInfo, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (info != 0) return fail(ctx, TCSCF_ERR_LINALG, "density eigen-decomposition failed");
  double lmax = 0;
  for (double v : hW) lmax = std::max(lmax, std::fabs(v));
  std::vector<int> hk;
  for (int e = nb - 1; e >= 0; --e)
    if (std::fabs(hW[e]) > 1e-12 * lmax) hk.push_back(e);
  int const nk = int(hk.size());
  if (nk == 0) { f.R = 0; return TCSCF_OK; }
  TCSCF_CUDA(ctx, cudaMemcpyAsync(keep, hk.data(), nk * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
  if (!f.complex) {
    kRealFactors<<<gridBlocks(int64_t(nb) * nk, 256), 256, 0, ctx->stream>>>(nb, nk, keep, W, A, f.ldx, f.X1, f.X2);
    f.R = nk;
  } else {
    kComplexFactors<<<gridBlocks(int64_t(nb) * nk, 256), 256, 0, ctx->stream>>>(nb, nk, keep, W, Z, f.ldx, f.X1, f.X1im, f.X2);
    f.R = 2 * nk;
  }
  TCSCF_LAUNCH(ctx);
  // host vectors go out of scope only after the stream has consumed `keep`
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

// Factor the spin density's real-harmonic form DR = X1 X2^T (one host synchronisation when the
// pivoted Cholesky factor applies; see factorFinish).
int factorDensity(tcscf_ctx * ctx, Grid & g, const double2 * dD, int spin, Factor & f)
{
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, spin ? "fac1" : "fac0", factorBufBytes(g.nb), &p));
  FactorBufs const b = carveFactorBufs(p, g.nb);
  TCSCF_TRY(factorLaunch(ctx, factorJob(g, dD, b), nullptr, 1, g.nb));
  FactorStatus st;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(&st, b.status, sizeof(FactorStatus), cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return factorFinish(ctx, g, b, st, f);
}

int checkBasisPair(tcscf_ctx * ctx, Grid * g1, Grid * g2)
{
  TCSCF_CHECK(ctx, g1 && g2, TCSCF_ERR_INVALID_ARGUMENT, "unknown grid handle");
  TCSCF_CHECK(ctx, g1->nb > 0 && g2->nb > 0, TCSCF_ERR_INVALID_ARGUMENT, "setBasisFunctions has not been called on the grid");
  TCSCF_CHECK(ctx, g1->nb == g2->nb, TCSCF_ERR_INVALID_ARGUMENT, "r1Grid.nBasis() != r2Grid.nBasis()");
  TCSCF_CHECK(ctx, g1->ndim == 3, TCSCF_ERR_INVALID_ARGUMENT, "the r1 grid must be three dimensional");
  for (int b = 0; b < g1->nb; ++b) {
    tcscf_sto const & a = g1->basis[b];
    tcscf_sto const & c = g2->basis[b];
    TCSCF_CHECK(ctx, a.alpha == c.alpha && a.n == c.n && a.l == c.l && a.m == c.m && a.family == c.family, TCSCF_ERR_INVALID_ARGUMENT,
                "r1 and r2 grids carry different basis sets");
  }
  return TCSCF_OK;
}

// Direct-form Fock build with device-resident densities dD [nspin][nb][nb] complex.
// Leaves G (masked), Fock (row-major) and the energy on the device.
int fockBuildDevice(tcscf_ctx * ctx, Grid & g1, Grid & g2, int nspin, const double2 * dD, const double * dH, int respectSym,
                    int precision, double2 * dG, double2 * dFock, double * dE, Factor const * given)
{
  int const nb = g1.nb;
  int64_t const n1 = g1.n, n2 = g2.n;
  double const scale = g2.ndim == 2 ? 2 * kPi : 1.0;
  int const ldt = nb;
  int const ldpsi = 2 * nb;
  size_t const bytes = sizeof(double) * (size_t(n2) * nb                 // V
                                         + size_t(n1) * ldpsi + size_t(n2) * ldpsi  // psi1, psi2
                                         + size_t(n2)                              // coul
                                         + size_t(nspin) * n1 * ldt                // T re
                                         + size_t(nspin) * n1 * ldt                // T im
                                         + size_t(nspin) * n1 + n1                 // VH per spin + total
                                         + size_t(nspin) * nb * nb * 2);           // GR re/im
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "fock", bytes, &p));
  double * V = static_cast<double *>(p);
  double * psi1 = V + size_t(n2) * nb;
  double * psi2 = psi1 + size_t(n1) * ldpsi;
  double * coul = psi2 + size_t(n2) * ldpsi;
  double * Tre = coul + n2;
  double * Tim = Tre + size_t(nspin) * n1 * ldt;
  double * VH = Tim + size_t(nspin) * n1 * ldt;
  double * VHtot = VH + size_t(nspin) * n1;
  double * GRre = VHtot + n1;
  double * GRim = GRre + size_t(nspin) * nb * nb;

  cudaEventRecord(ctx->ev[0], ctx->stream);
  int const launch0 = ctx->launchCount;
  int nparts = 0, symSpin = 0, complexSpin = 0;
  double const * Vdone = nullptr;   // V once a spin has formed it
  const void * vtPacked = nullptr;
  for (int s = 0; s < nspin; ++s) {
    Factor f;
    if (given && given[s].X1) f = given[s];   // the caller's factor of this spin's density (its occupied orbitals)
    else TCSCF_TRY(factorDensity(ctx, g1, dD + size_t(s) * nb * nb, s, f));
    double * Ts = Tre + size_t(s) * n1 * ldt;
    double * Ti = Tim + size_t(s) * n1 * ldt;
    if (f.R == 0) {
      TCSCF_CUDA(ctx, cudaMemsetAsync(Ts, 0, sizeof(double) * n1 * ldt, ctx->stream));
      TCSCF_CUDA(ctx, cudaMemsetAsync(VH + size_t(s) * n1, 0, sizeof(double) * n1, ctx->stream));
      continue;
    }
    int const R = f.R;
    // one grid on both sides and X1 = X2: psi1 = psi2 and X = g rho is symmetric, so the split-BF16 and
    // FP64 contractions compute only the pairs on and above each r1 tile's diagonal (T'), and the
    // exchange matrix is sum W T' plus its transpose (TF32 keeps the full form: tensorPrepare)
    bool const sym = precision != TCSCF_PREC_TF32 && &g1 == &g2 && f.same;
    if (sym) symSpin |= 1 << s;
    if (f.complex) complexSpin |= 1 << s;
    for (int part = 0; part < (f.complex ? 2 : 1); ++part) {
      double const * X1 = part == 0 ? f.X1 : f.X1im;
      OrbitalArgs o1{n1, nb, R, f.ldx, ldpsi, 0, 0, scale, g1.phiR, g1.w, X1, nullptr, psi1, nullptr, nullptr};
      // the r2 side (the r1 side where the two are one): psi2, the Coulomb source with the r1-side factor on
      // the r2 points (rho(r2, r2)), and V for the first spin
      OrbitalArgs o2 = o1;
      o2.n = n2; o2.phi = g2.phiR; o2.w = g2.w; o2.coul = coul;
      o2.V = Vdone ? nullptr : V;
      if (sym) TCSCF_TRY(orbitals(ctx, o2));
      else {
        TCSCF_TRY(orbitals(ctx, o1));
        o2.X = f.X2; o2.Xc = f.same ? nullptr : f.X1; o2.psi = psi2;
        if (part == 0) TCSCF_TRY(orbitals(ctx, o2));
      }
      Vdone = V;
      if (precision == TCSCF_PREC_BF16X3 && !vtPacked) TCSCF_TRY(tensorPackedV(ctx, g2, V, scale, &vtPacked));
      double const * p2side = sym ? psi1 : psi2;
      Contraction c;
      c.n1 = n1; c.n2 = n2; c.R = R; c.ncol = nb;
      c.p1 = g1.pts; c.p2 = g2.pts; c.psi1 = psi1; c.psi2 = p2side; c.ldpsi = ldpsi;
      c.V = V; c.ldv = nb; c.T = part == 0 ? Ts : Ti; c.ldt = ldt;
      c.vtPacked = vtPacked;
      c.sym = sym ? 1 : 0;
      if (precision != TCSCF_PREC_FP64) TCSCF_TRY(nearPairsFor(ctx, g1, g2, &c.near));
      if (part == 0) {
        c.coul = coul;
        c.VH = VH + size_t(s) * n1;
      }
      // the contraction routines bracket their main kernel with evStart() / evStop()
      ctx->evPart = nparts++;
      int const st = precision == TCSCF_PREC_FP64 ? contractFp64(ctx, c) : contractTensor(ctx, c, precision);
      ctx->evPart = 0;
      TCSCF_TRY(st);
    }
  }
  if (nspin == 2) {
    kAddSpins<<<gridBlocks(n1, 256), 256, 0, ctx->stream>>>(n1, VH, VH + n1, VHtot);
    TCSCF_LAUNCH(ctx);
  }
  double const * potential = nspin == 2 ? VHtot : VH;
  // a symmetric spin's G is M + M^T of the sums over T', with the (symmetric) Coulomb part at half weight in M
  double const cJ0 = nspin == 1 ? 2.0 : 1.0;
  double const cJ[2] = {symSpin & 1 ? 0.5 * cJ0 : cJ0, symSpin & 2 ? 0.5 * cJ0 : cJ0};
  TCSCF_TRY(reduceFockReal(ctx, n1, nb, nspin, g1.phiR, g1.w, potential, cJ, Tre, int64_t(n1) * ldt, ldt, GRre));
  if (complexSpin) {
    double const none[2] = {0.0, 0.0};
    for (int s = 0; s < nspin; ++s)
      if (!((complexSpin >> s) & 1)) TCSCF_CUDA(ctx, cudaMemsetAsync(Tim + size_t(s) * n1 * ldt, 0, sizeof(double) * n1 * ldt, ctx->stream));
    TCSCF_TRY(reduceFockReal(ctx, n1, nb, nspin, g1.phiR, g1.w, nullptr, none, Tim, int64_t(n1) * ldt, ldt, GRim));
  }
  ctx->lastVH = potential;
  ctx->lastT = Tre;
  ctx->lastN1 = n1;
  ctx->lastNb = nb;
  TCSCF_TRY(fockFinish(ctx, nspin, nb, {GRre, complexSpin ? GRim : nullptr, g1.dsto, symSpin}, dH, dG, nullptr, dD, respectSym, cJ0, dFock, dE));
  cudaEventRecord(ctx->ev[1], ctx->stream);
  TCSCF_CUDA(ctx, cudaEventSynchronize(ctx->ev[1]));
  float tot = 0;
  cudaEventElapsedTime(&tot, ctx->ev[0], ctx->ev[1]);
  double contractionMs = 0;
  for (int k = 0; k < nparts; ++k) {
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx->ev[2 + 2 * k], ctx->ev[3 + 2 * k]);
    contractionMs += ms;
  }
  ctx->lastTotalMs = tot;
  ctx->lastContractionMs = contractionMs;
  ctx->lastLaunches = ctx->launchCount - launch0;
  return TCSCF_OK;
}

// Batched RCS Fock builds (tcscf_fock_build_batch): every instance's density is factored and its
// tensor operands packed into its own arena; then all tensor contractions run in one persistent
// launch per tile class, and each instance's Fock matrix and energy are finished.  Instances whose
// density factor is complex in the real-harmonic basis, or whose shape the tensor path does not
// take, are built on their own with fockBuildDevice.
int fockBuildBatch(tcscf_ctx * ctx, int count, Grid * const * g1s, Grid * const * g2s, const double2 * const * dDs, const double * const * dHs,
                   int respectSym, int precision, double2 * const * dGs, double2 * const * dFs, double * const * dEs)
{
  cudaEventRecord(ctx->ev[0], ctx->stream);
  int const launch0 = ctx->launchCount;
  // shared temporaries (consumed in stream order by each instance's packing before the next reuses them)
  int64_t maxN1 = 0, maxN2 = 0;
  int maxNb = 0;
  for (int k = 0; k < count; ++k) {
    maxN1 = std::max(maxN1, g1s[k]->n);
    maxN2 = std::max(maxN2, g2s[k]->n);
    maxNb = std::max(maxNb, g1s[k]->nb);
  }
  size_t const tmpBytes = sizeof(double) * (2 * size_t(maxN2) * maxNb + size_t(maxN1) * maxNb + size_t(maxN2));
  void * tp = nullptr;
  TCSCF_TRY(scratch(ctx, "batch_tmp", tmpBytes, &tp));
  double * V = static_cast<double *>(tp);
  double * psi1 = V + size_t(maxN2) * maxNb;
  double * psi2 = psi1 + size_t(maxN1) * maxNb;
  double * coul = psi2 + size_t(maxN2) * maxNb;

  // per-instance persistent buffers: T, VH, GR and the tensor arena
  std::vector<Contraction> cs(count);
  std::vector<char> tensorOk(count, 0);
  std::vector<size_t> offs(count + 1, 0);
  std::vector<size_t> arenaBytes(count, 0);
  for (int k = 0; k < count; ++k) {
    Grid & g1 = *g1s[k];
    Grid & g2 = *g2s[k];
    int const nb = g1.nb;
    Contraction & c = cs[k];
    c.n1 = g1.n; c.n2 = g2.n; c.R = std::min(nb, 32); c.ncol = nb; c.ldpsi = nb; c.ldt = nb;
    c.p1 = g1.pts; c.p2 = g2.pts;
    c.nSplit = splitForPolicy(c, precision, ctx->batchSplitPolicy);
    arenaBytes[k] = tensorArenaBytes(c, precision);
    size_t const own = (sizeof(double) * (size_t(g1.n) * nb + g1.n + size_t(nb) * nb) + 255) & ~size_t(255);
    offs[k + 1] = offs[k] + own + ((arenaBytes[k] + 255) & ~size_t(255));
  }
  void * bp = nullptr;
  TCSCF_TRY(scratch(ctx, "batch_arena", offs[count] + 256, &bp));
  // every instance's density is factored in one launch (a block each), with one host synchronisation for all
  std::vector<size_t> fOffs(count + 1, 0);
  for (int k = 0; k < count; ++k) fOffs[k + 1] = fOffs[k] + ((factorBufBytes(g1s[k]->nb) + 255) & ~size_t(255));
  void * fp = nullptr;
  TCSCF_TRY(scratch(ctx, "batch_factors", fOffs[count] + 256, &fp));
  size_t const jobBytes = (sizeof(FactorJob) * count + 255) & ~size_t(255);
  void * sp = nullptr;
  TCSCF_TRY(scratch(ctx, "batch_factor_status", jobBytes + sizeof(FactorStatus) * count + 256, &sp));
  auto * dJobs = static_cast<FactorJob *>(sp);
  auto * dStatus = reinterpret_cast<FactorStatus *>(static_cast<char *>(sp) + jobBytes);
  std::vector<FactorBufs> fbufs(count);
  std::vector<FactorJob> jobs(count);
  for (int k = 0; k < count; ++k) {
    fbufs[k] = carveFactorBufs(static_cast<char *>(fp) + fOffs[k], g1s[k]->nb);
    fbufs[k].status = dStatus + k;
    jobs[k] = factorJob(*g1s[k], dDs[k], fbufs[k]);
  }
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dJobs, jobs.data(), sizeof(FactorJob) * count, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_TRY(factorLaunch(ctx, FactorJob{}, dJobs, count, maxNb));
  std::vector<FactorStatus> hStatus(count);
  TCSCF_CUDA(ctx, cudaMemcpyAsync(hStatus.data(), dStatus, sizeof(FactorStatus) * count, cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::vector<TensorPrep> preps(count);
  std::vector<TensorPrep *> ready;
  for (int k = 0; k < count; ++k) {
    Grid & g1 = *g1s[k];
    Grid & g2 = *g2s[k];
    int const nb = g1.nb;
    int64_t const n1 = g1.n, n2 = g2.n;
    double const scale = g2.ndim == 2 ? 2 * kPi : 1.0;
    char * base = static_cast<char *>(bp) + offs[k];
    double * T = reinterpret_cast<double *>(base);
    double * VH = T + size_t(n1) * nb;   // followed by the instance's [nb][nb] reduction output
    void * arena = base + ((sizeof(double) * (size_t(n1) * nb + n1 + size_t(nb) * nb) + 255) & ~size_t(255));
    Factor f;
    TCSCF_TRY(factorFinish(ctx, g1, fbufs[k], hStatus[k], f));
    Contraction & c = cs[k];
    // one grid on both sides and X1 = X2: the symmetric split-BF16 contraction (psi2 = psi1)
    bool const sym = precision == TCSCF_PREC_BF16X3 && &g1 == &g2 && f.same;
    c.R = f.R;
    c.T = T; c.VH = VH; c.V = V; c.ldv = nb;
    c.psi1 = psi1; c.psi2 = sym ? psi1 : psi2; c.coul = coul;
    c.sym = sym ? 1 : 0;
    std::string why;
    bool eligible = (precision == TCSCF_PREC_BF16X3 || precision == TCSCF_PREC_TF32) && f.R > 0 && !f.complex &&
                    tensorPathAvailable(c, precision, &why) && tensorArenaBytes(c, precision) <= arenaBytes[k];
    if (eligible) {
      // an instance whose grids hold near-coincident pairs is built on its own (with the FP64 correction)
      NearList const * nl = nullptr;
      TCSCF_TRY(nearPairsFor(ctx, g1, g2, &nl));
      eligible = nl->count == 0;
    }
    if (!eligible) continue;
    OrbitalArgs o1{n1, nb, f.R, f.ldx, nb, 0, 0, scale, g1.phiR, g1.w, f.X1, nullptr, psi1, nullptr, nullptr};
    OrbitalArgs o2 = o1;
    o2.n = n2; o2.phi = g2.phiR; o2.w = g2.w; o2.coul = coul; o2.V = V;
    if (!sym) {
      TCSCF_TRY(orbitals(ctx, o1));
      o2.X = f.X2; o2.Xc = f.same ? nullptr : f.X1; o2.psi = psi2;
    }
    TCSCF_TRY(orbitals(ctx, o2));
    const void * vtPacked = nullptr;
    if (precision == TCSCF_PREC_BF16X3) TCSCF_TRY(tensorPackedV(ctx, g2, V, scale, &vtPacked));
    c.vtPacked = vtPacked;
    TCSCF_TRY(tensorPrepare(ctx, c, precision, arena, arenaBytes[k], preps[k]));
    tensorOk[k] = 1;
    ready.push_back(&preps[k]);
  }
  if (!ready.empty()) TCSCF_TRY(tensorRun(ctx, ready.data(), int(ready.size())));
  float contractionMs = 0;
  if (!ready.empty()) {
    TCSCF_CUDA(ctx, cudaEventSynchronize(ctx->evStop()));
    cudaEventElapsedTime(&contractionMs, ctx->evStart(), ctx->evStop());
  }
  for (int k = 0; k < count; ++k) {
    Grid & g1 = *g1s[k];
    int const nb = g1.nb;
    if (!tensorOk[k]) {
      TCSCF_TRY(fockBuildDevice(ctx, g1, *g2s[k], 1, dDs[k], dHs[k], respectSym, precision, dGs[k], dFs[k], dEs[k], nullptr));
      continue;
    }
    Contraction const & c = cs[k];
    double * GR = c.VH + g1.n;
    double const cJ[2] = {c.sym ? 1.0 : 2.0, 0.0};
    TCSCF_TRY(reduceFockReal(ctx, g1.n, nb, 1, g1.phiR, g1.w, c.VH, cJ, c.T, 0, nb, GR));
    TCSCF_TRY(fockFinish(ctx, 1, nb, {GR, nullptr, g1.dsto, c.sym}, dHs[k], dGs[k], nullptr, dDs[k], respectSym, 2.0, dFs[k], dEs[k]));
  }
  cudaEventRecord(ctx->ev[1], ctx->stream);
  TCSCF_CUDA(ctx, cudaEventSynchronize(ctx->ev[1]));
  float tot = 0;
  cudaEventElapsedTime(&tot, ctx->ev[0], ctx->ev[1]);
  ctx->lastTotalMs = tot;
  ctx->lastContractionMs = contractionMs;
  ctx->lastLaunches = ctx->launchCount - launch0;
  return TCSCF_OK;
}

int validateBasis(tcscf_ctx * ctx, const tcscf_sto * basis, int nb, std::vector<DevSto> & out)
{
  TCSCF_CHECK(ctx, basis && nb > 0, TCSCF_ERR_INVALID_ARGUMENT, "empty basis");
  out.resize(nb);
  for (int b = 0; b < nb; ++b) {
    tcscf_sto const & s = basis[b];
    TCSCF_CHECK(ctx, s.family == basis[0].family, TCSCF_ERR_INVALID_ARGUMENT, "a basis holds one family of functions");
    TCSCF_CHECK(ctx, s.l <= kMaxL, TCSCF_ERR_UNSUPPORTED, "angular momentum above 12");
    TCSCF_CHECK(ctx, s.l >= std::abs(s.m), TCSCF_ERR_INVALID_ARGUMENT, "|m| > l");
    if (s.family == TCSCF_BASIS_STO) {
      // SlaterTypeOrbital.hpp:34-36
      TCSCF_CHECK(ctx, s.n >= 1 && s.n >= s.l, TCSCF_ERR_INVALID_ARGUMENT, "invalid STO quantum numbers");
      TCSCF_CHECK(ctx, s.alpha > 0, TCSCF_ERR_INVALID_ARGUMENT, "non-positive STO exponent");
    } else if (s.family == TCSCF_BASIS_OCHI) {
      // OchiBasis.hpp:33-34
      TCSCF_CHECK(ctx, s.n >= 0, TCSCF_ERR_INVALID_ARGUMENT, "negative Ochi Laguerre degree");
      TCSCF_CHECK(ctx, s.alpha > 0, TCSCF_ERR_INVALID_ARGUMENT, "non-positive Ochi exponent");
    } else if (s.family == TCSCF_BASIS_HYDROGEN) {
      // HydrogenLikeBasis.hpp:31-34
      TCSCF_CHECK(ctx, s.alpha > 0 && s.n >= 1 && s.l < s.n, TCSCF_ERR_INVALID_ARGUMENT, "invalid hydrogen-like quantum numbers or Z");
    } else {
      return fail(ctx, TCSCF_ERR_INVALID_ARGUMENT, "unknown basis family");
    }
    DevSto d{};
    d.alpha = s.family == TCSCF_BASIS_HYDROGEN ? s.alpha / s.n : s.alpha;
    d.norm = basisNormalization(s);
    d.n = s.n; d.l = s.l; d.m = s.m;
    d.family = s.family;
    d.rtype = s.m == 0 ? 0 : (s.m > 0 ? 1 : 2);
    d.partner = -1;
    if (s.m != 0) {
      for (int c = 0; c < nb; ++c)
        if (basis[c].alpha == s.alpha && basis[c].n == s.n && basis[c].l == s.l && basis[c].m == -s.m && basis[c].family == s.family) {
          d.partner = c;
          break;
        }
      TCSCF_CHECK(ctx, d.partner >= 0, TCSCF_ERR_UNSUPPORTED, "basis lacks the -m partner of an m != 0 function");
    }
    out[b] = d;
  }
  return TCSCF_OK;
}

// precomputeIntegrand + computeF / computeV (HartreeFock.hpp:23-229): the weighted basis-pair products
// of the r2 grid (real-harmonic basis, k <= l) contracted with the r12 kernel (ncomp = 1: a scalar
// kernel; 3: the components of grad_1 u) in the requested precision, then mapped to the reference's
// complex Fji / Vji layout; written to host memory (out) and / or kept on the device as a handle.
int precomputeTensor(tcscf_ctx * ctx, int r1, int r2, int kernel, const tcscf_ochi * jastrow, int precision, int ncomp, double * out,
                     int keep, int * handle)
{
  Grid * g1 = findGrid(ctx, r1);
  Grid * g2 = findGrid(ctx, r2);
  TCSCF_TRY(checkBasisPair(ctx, g1, g2));
  TCSCF_CHECK(ctx, !jastrow || (jastrow->nterms >= 0 && jastrow->nterms <= 8), TCSCF_ERR_INVALID_ARGUMENT, "at most 8 Jastrow terms");
  TCSCF_CHECK(ctx, out || keep, TCSCF_ERR_INVALID_ARGUMENT, "nothing to do");
  TCSCF_CHECK(ctx, ncomp == 1 || g2->ndim == 3, TCSCF_ERR_INVALID_ARGUMENT, "computeV needs a 3-D r2 grid");
  TCSCF_CHECK(ctx, precision == TCSCF_PREC_FP64 || precision == TCSCF_PREC_BF16X3, TCSCF_ERR_UNSUPPORTED,
              "computeF / computeV run in FP64 or BF16X3");
  int const nb = g1->nb;
  int const np = nb * (nb + 1) / 2;
  int64_t const n1 = g1->n, n2 = g2->n;
  bool const realOut = ncomp == 1 && g2->ndim == 2;
  double const scale = realOut ? 2 * kPi : 1.0;
  Contraction c;
  c.n1 = n1; c.n2 = n2; c.R = 0; c.ncol = np; c.p1 = g1->pts; c.p2 = g2->pts; c.ldv = np; c.ldt = np;
  c.kernel = kernel; c.jastrow = jastrow;
  if (precision != TCSCF_PREC_FP64) {
    std::string why;
    TCSCF_CHECK(ctx, pairsTensorAvailable(c, precision, &why), TCSCF_ERR_UNSUPPORTED, why);
    TCSCF_TRY(nearPairsFor(ctx, *g1, *g2, &c.near));
  }
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "computeF", sizeof(double) * (size_t(n2) * np + size_t(n1) * np), &p));
  double * pairs = static_cast<double *>(p);
  double * FR = pairs + size_t(n2) * np;
  Tensor t;
  t.n1 = n1; t.nb = nb; t.isComplex = realOut ? 0 : 1; t.vec = ncomp == 3 ? 1 : 0;
  TCSCF_TRY(tensorAlloc(ctx, t, sizeof(double) * size_t(n1) * ncomp * tensorPlane(nb)));
  cudaEventRecord(ctx->ev[0], ctx->stream);
  int const launch0 = ctx->launchCount;
  kPairProducts<<<gridBlocks(n2 * np, 256), 256, 0, ctx->stream>>>(n2, nb, g2->phiR, g2->w, scale, pairs);
  ctx->launchCount++;
  int st = TCSCF_OK;
  if (cudaError_t const e = cudaGetLastError(); e != cudaSuccess)   // the tensor is released below
    st = fail(ctx, TCSCF_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
  c.V = pairs;
  c.T = FR;
  for (int comp = 0; comp < ncomp && st == TCSCF_OK; ++comp) {
    c.component = comp;
    // the contractions alone are bracketed by evStart() / evStop(); tcscf_last_timing reports the components' sum
    ctx->evPart = comp;
    cudaEventRecord(ctx->evStart(), ctx->stream);
    st = precision == TCSCF_PREC_FP64 ? contractFp64(ctx, c) : contractPairsTensor(ctx, c, precision);
    cudaEventRecord(ctx->evStop(), ctx->stream);
    if (st == TCSCF_OK) {
      kPairsToPlanes<<<gridBlocks(n1 * tensorPlane(nb), 256), 256, 0, ctx->stream>>>(n1, nb, FR, ncomp, comp, t.d);
      ctx->launchCount++;
      cudaError_t const e = cudaGetLastError();
      if (e != cudaSuccess) st = fail(ctx, TCSCF_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  ctx->evPart = 0;
  if (st == TCSCF_OK && out) {
    // the reference layout for the host, in pieces of at most 1 GiB
    size_t const row = sizeof(double) * size_t(nb) * nb * ncomp * (realOut ? 1 : 2);
    int64_t const chunk = std::max<int64_t>(1, std::min<int64_t>(n1, int64_t((size_t(1) << 30) / row)));
    void * q = nullptr;
    st = scratch(ctx, "tensor_out", row * chunk, &q);
    for (int64_t r0 = 0; r0 < n1 && st == TCSCF_OK; r0 += chunk) {
      int64_t const rows = std::min(chunk, n1 - r0);
      st = tensorToReference(ctx, t, g1->dsto, r0, rows, static_cast<double *>(q));
      cudaError_t const e = st == TCSCF_OK ? cudaMemcpyAsync(reinterpret_cast<char *>(out) + row * r0, q, row * rows, cudaMemcpyDeviceToHost, ctx->stream)
                                           : cudaSuccess;
      if (e != cudaSuccess) st = fail(ctx, TCSCF_ERR_CUDA, cudaGetErrorString(e));
    }
  }
  cudaEventRecord(ctx->ev[1], ctx->stream);
  cudaStreamSynchronize(ctx->stream);
  float contraction = 0, b = 0;
  for (int comp = 0; comp < ncomp; ++comp) {
    float a = 0;
    if (st == TCSCF_OK) cudaEventElapsedTime(&a, ctx->ev[2 + 2 * comp], ctx->ev[3 + 2 * comp]);
    contraction += a;
  }
  cudaEventElapsedTime(&b, ctx->ev[0], ctx->ev[1]);
  ctx->lastContractionMs = contraction;
  ctx->lastTotalMs = b;
  ctx->lastLaunches = ctx->launchCount - launch0;
  if (st != TCSCF_OK || !keep) { tensorRelease(ctx, t); return st; }
  int const id = ctx->nextId++;
  ctx->tensors[id] = t;
  if (handle) *handle = id;
  return TCSCF_OK;
}

// ---- SCF as one CUDA graph (tcscf_scf_graph) ------------------------------------------------------
// C = op(A) B for small dense row-major matrices (op(A) = A [M][K] or A^T with A [K][M]); one thread
// per output element
__global__ void kSmallGemm(int M, int N, int K, const double * A, int lda, int transA, const double * B, int ldb, double * C, int ldc)
{
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < M * N; idx += gridDim.x * blockDim.x) {
    int const i = idx / N, j = idx % N;
    double s = 0;
    for (int k = 0; k < K; ++k) s = fma(transA ? A[k * lda + i] : A[i * lda + k], B[k * ldb + j], s);
    C[i * ldc + j] = s;
  }
}

// Two-sided cyclic Jacobi eigen-solver of the symmetric m x m matrix A (row-major) in one CTA
// (Golub & Van Loan, Matrix Computations, sym.schur2 rotations in the round-robin parallel ordering:
// m (rounded up to even, the padding index carries a zero row) indices are paired into m/2 disjoint
// rotations per step, m - 1 steps per sweep).  A lives in shared memory, the eigenvectors V (columns,
// row-major [m][m]) in global memory.  A rotation is skipped when |a_pq| <= eps sqrt|a_pp a_qq|; the
// sweeps stop when one performs no rotation (at most 40).  Out: W[m] the eigenvalues (A's diagonal,
// unsorted) and V.
constexpr int kJacobiThreads = 512;
__global__ void __launch_bounds__(kJacobiThreads) kJacobiSym(int m, const double * Ain, double * W, double * V)
{
  extern __shared__ double sJ[];
  __shared__ double cs[64], sn[64];
  __shared__ int pp[64], qq[64];
  __shared__ int rotated;
  int const mp = m + (m & 1);
  int const half = mp / 2;
  int const tid = threadIdx.x;
  for (int idx = tid; idx < mp * mp; idx += blockDim.x) {
    int const i = idx / mp, j = idx % mp;
    sJ[idx] = (i < m && j < m) ? 0.5 * (Ain[i * m + j] + Ain[j * m + i]) : 0.0;
  }
  for (int idx = tid; idx < m * m; idx += blockDim.x) V[idx] = (idx / m == idx % m) ? 1.0 : 0.0;
  __syncthreads();
  for (int sweep = 0; sweep < 40; ++sweep) {
    if (tid == 0) rotated = 0;
    __syncthreads();
    for (int step = 0; step < mp - 1; ++step) {
      if (tid < half) {
        // round-robin pairing: index mp - 1 stays, the others rotate by one each step
        int p = tid == 0 ? mp - 1 : (step + tid) % (mp - 1);
        int q = (step + mp - 1 - tid) % (mp - 1);
        if (tid == 0) q = step % (mp - 1);
        if (p > q) { int const t = p; p = q; q = t; }
        double const apq = sJ[p * mp + q], app = sJ[p * mp + p], aqq = sJ[q * mp + q];
        double c = 1.0, s = 0.0;
        if (apq != 0.0 && fabs(apq) > 2.2204460492503131e-16 * sqrt(fabs(app * aqq))) {
          double const tau = (aqq - app) / (2.0 * apq);
          double const t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
          c = 1.0 / sqrt(1.0 + t * t);
          s = t * c;
          rotated = 1;
        }
        pp[tid] = p; qq[tid] = q; cs[tid] = c; sn[tid] = s;
      }
      __syncthreads();
      // rows: A <- J^T A
      for (int idx = tid; idx < half * mp; idx += blockDim.x) {
        int const k = idx / mp, j = idx % mp;
        if (sn[k] == 0.0) continue;
        int const p = pp[k], q = qq[k];
        double const c = cs[k], s = sn[k];
        double const ap = sJ[p * mp + j], aq = sJ[q * mp + j];
        sJ[p * mp + j] = c * ap - s * aq;
        sJ[q * mp + j] = s * ap + c * aq;
      }
      __syncthreads();
      // columns: A <- A J, V <- V J
      for (int idx = tid; idx < half * mp; idx += blockDim.x) {
        int const k = idx / mp, i = idx % mp;
        if (sn[k] == 0.0) continue;
        int const p = pp[k], q = qq[k];
        double const c = cs[k], s = sn[k];
        double const ap = sJ[i * mp + p], aq = sJ[i * mp + q];
        sJ[i * mp + p] = c * ap - s * aq;
        sJ[i * mp + q] = s * ap + c * aq;
        if (i < m && q < m) {
          double const vp = V[i * m + p], vq = V[i * m + q];
          V[i * m + p] = c * vp - s * vq;
          V[i * m + q] = s * vp + c * vq;
        }
      }
      __syncthreads();
    }
    if (!rotated) break;
    __syncthreads();
  }
  for (int i = tid; i < m; i += blockDim.x) W[i] = sJ[i * mp + i];
}

// Eigenvalues in ascending order (ties by index): Ws[m], and the indices of the nocc lowest; then
// the occupied coefficients C[k][a] = sum_j Xc[k][j] V[j][idx[a]] ([nb][nocc], real-harmonic basis)
// and the density DR = C C^T.  One block.
__global__ void kOccupiedOrbitals(int nb, int m, int nocc, const double * W, const double * V, const double * Xc, double * Ws, double * C,
                                  double * DR)
{
  __shared__ int idx[128];
  for (int t = threadIdx.x; t < m; t += blockDim.x) {
    double const wt = W[t];
    int r = 0;
    for (int j = 0; j < m; ++j) r += (W[j] < wt || (W[j] == wt && j < t)) ? 1 : 0;
    Ws[r] = wt;
    if (r < nocc) idx[r] = t;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nb * nocc; e += blockDim.x) {
    int const k = e / nocc, a = e % nocc;
    double s = 0;
    for (int j = 0; j < m; ++j) s = fma(Xc[k * m + j], V[j * m + idx[a]], s);
    C[e] = s;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nb * nb; e += blockDim.x) {
    int const u = e / nb, v = e % nb;
    double s = 0;
    for (int a = 0; a < nocc; ++a) s = fma(C[u * nocc + a], C[v * nocc + a], s);
    DR[e] = s;
  }
}

// The convergence test of the SCF loop (RCSHartreeFock::compute, HartreeFock.cpp:857): the energy of
// this iteration's build against the previous one; on convergence, a non-finite energy, an expired
// bounded wait of the tensor kernel or the iteration limit, the loop ends (the graph's WHILE
// condition is cleared) with the density and eigenvalues this build used saved.
struct ScfGraphState {
  double eprev, eres;
  int iter, done, code, pad;
};
__global__ void kScfCheck(ScfGraphState * st, const double * E, const int * tstatus, int maxIter, double tol, int nD, const double2 * D,
                          double2 * Dres, int nW, const double * Wcur, double * Wres, cudaGraphConditionalHandle handle, int useHandle)
{
  __shared__ int stop;
  if (threadIdx.x == 0) {
    double const e = *E;
    int const it = st->iter + 1;
    st->iter = it;
    int code = TCSCF_OK;
    bool s = true;
    if (tstatus && *tstatus != 0) code = TCSCF_ERR_TIMEOUT;
    else if (!isfinite(e)) code = TCSCF_ERR_NONFINITE;
    else if (fabs(e - st->eprev) < tol) code = TCSCF_OK;
    else if (it >= maxIter) code = TCSCF_ERR_NOT_CONVERGED;
    else s = false;
    st->eprev = e;
    if (s) { st->done = 1; st->code = code; st->eres = e; }
    stop = s ? 1 : 0;
  }
  __syncthreads();
  if (stop) {
    for (int i = threadIdx.x; i < nD; i += blockDim.x) Dres[i] = D[i];
    for (int i = threadIdx.x; i < nW; i += blockDim.x) Wres[i] = Wcur[i];
  }
  if (useHandle && threadIdx.x == 0) cudaGraphSetConditional(handle, stop ? 0u : 1u);
}

// One RCS SCF on the device (tcscf_scf_graph).  Every iteration is the same launch sequence on fixed
// buffers: orbitals of the current occupied coefficients C on both grids, the Coulomb source, the r12
// contraction (FP64 or tensor cores) from those factors (D = C C^T, rank nocc), the real Fock
// reduction, the reference-basis G, F and energy (kFockFinish), the convergence test, then the new C from
// the Fock matrix: real-harmonic F, Xc^T F Xc with the canonical orthogonaliser Xc of S, Jacobi, the
// nocc lowest eigenvectors.  The first two iterations run directly (the zero-density one, F = h, with
// no contraction; the second allocates every buffer); with capture the rest run as one graph launch
// whose conditional WHILE node repeats the body until the device-side test clears it, so the host
// neither reads nor waits per iteration.
int scfGraph(tcscf_ctx * ctx, Grid & g1, Grid & g2, int nocc, const double * S, const double * h, int respectSym, int precision, double tol,
             int maxIter, int capture, double * energy, int * iterations, double * density, double * eigenvalues, int * graphLaunches)
{
  int const nb = g1.nb;
  int64_t const n1 = g1.n, n2 = g2.n;
  size_t const nn = size_t(nb) * nb;
  double const scale = g2.ndim == 2 ? 2 * kPi : 1.0;
  TCSCF_CHECK(ctx, nb <= 128, TCSCF_ERR_UNSUPPORTED, "the graph SCF's device eigen-solver takes nb <= 128");
  TCSCF_CHECK(ctx, nocc >= 1 && nocc <= nb, TCSCF_ERR_INVALID_ARGUMENT, "occupied orbitals out of range");
  // ---- small buffers
  void * p = nullptr;
  size_t const smallBytes = sizeof(double2) * nn * 7 + sizeof(double) * (nn * 8 + size_t(nb) * nocc + 4 * nb + 64) + sizeof(ScfGraphState) + 4096;
  TCSCF_TRY(scratch(ctx, "scf_graph_small", smallBytes, &p));
  char * q = static_cast<char *>(p);
  auto take = [&](size_t n) { char * r = q; q += (n + 255) & ~size_t(255); return r; };
  auto * dD = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  auto * dG = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  auto * dF = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  auto * FRc = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  auto * Sc = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  auto * SRc = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  auto * Dres = reinterpret_cast<double2 *>(take(sizeof(double2) * nn));
  double * dH = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * FR = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * SR = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * Xc = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * Tm = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * Fp = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * Vm = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * DR = reinterpret_cast<double *>(take(sizeof(double) * nn));
  double * C = reinterpret_cast<double *>(take(sizeof(double) * nb * nocc));
  double * W = reinterpret_cast<double *>(take(sizeof(double) * nb));
  double * Ws = reinterpret_cast<double *>(take(sizeof(double) * nb));
  double * Wres = reinterpret_cast<double *>(take(sizeof(double) * nb));
  double * fmaxv = reinterpret_cast<double *>(take(sizeof(double) * 4));
  double * dE = reinterpret_cast<double *>(take(sizeof(double) * 4));
  auto * st = reinterpret_cast<ScfGraphState *>(take(sizeof(ScfGraphState)));
  // ---- grid-sized buffers of the build
  int const ldpsi = nocc;
  size_t const bigBytes = sizeof(double) * (size_t(n2) * nb + size_t(n1) * ldpsi + size_t(n2) * ldpsi + n2 + size_t(n1) * nb + n1) + 8 * 256;
  TCSCF_TRY(scratch(ctx, "scf_graph_build", bigBytes, &p));
  q = static_cast<char *>(p);
  double * Vw = reinterpret_cast<double *>(take(sizeof(double) * n2 * nb));
  double * psi1 = reinterpret_cast<double *>(take(sizeof(double) * n1 * ldpsi));
  double * psi2 = reinterpret_cast<double *>(take(sizeof(double) * n2 * ldpsi));
  double * coul = reinterpret_cast<double *>(take(sizeof(double) * n2));
  double * Tb = reinterpret_cast<double *>(take(sizeof(double) * n1 * nb));
  double * VH = reinterpret_cast<double *>(take(sizeof(double) * n1));

  // ---- canonical orthogonaliser Xc = U s^-1/2 of the real-harmonic overlap (eigenvalues above 1e-12
  // of the largest kept)
  TCSCF_CUDA(ctx, cudaMemcpyAsync(SR, S, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dH, h, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  kRealToComplex<<<gridBlocks(int64_t(nn), 256), 256, 0, ctx->stream>>>(int64_t(nn), SR, Sc);
  TCSCF_LAUNCH(ctx);
  kDensityToReal<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, g1.dsto, Sc, SRc);
  TCSCF_LAUNCH(ctx);
  kSplitDensity<<<1, 256, 0, ctx->stream>>>(nb, SRc, SR, fmaxv);
  TCSCF_LAUNCH(ctx);
  int m = 0;
  {
    int lwork = 0;
    if (cusolverDnDsyevd_bufferSize(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, nb, SR, nb, W, &lwork) != CUSOLVER_STATUS_SUCCESS)
      return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnDsyevd_bufferSize failed");
    void * wk = nullptr;
    TCSCF_TRY(scratch(ctx, "scf_graph_syevd", sizeof(double) * size_t(lwork) + 64 + sizeof(int) * 4, &wk));
    int * info = reinterpret_cast<int *>(static_cast<double *>(wk) + lwork);
    if (cusolverDnDsyevd(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, nb, SR, nb, W, static_cast<double *>(wk), lwork, info) !=
        CUSOLVER_STATUS_SUCCESS)
      return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnDsyevd failed");
    std::vector<double> hs(nb), hv(nn);
    int hinfo = 0;
    TCSCF_CUDA(ctx, cudaMemcpyAsync(hs.data(), W, sizeof(double) * nb, cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaMemcpyAsync(hv.data(), SR, sizeof(double) * nn, cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaMemcpyAsync(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    TCSCF_CHECK(ctx, hinfo == 0 && hs[nb - 1] > 0 && std::isfinite(hs[nb - 1]), TCSCF_ERR_LINALG, "overlap matrix is not positive definite");
    std::vector<int> keep;
    for (int j = 0; j < nb; ++j)
      if (hs[j] > 1e-12 * hs[nb - 1]) keep.push_back(j);
    m = int(keep.size());
    TCSCF_CHECK(ctx, m >= nocc, TCSCF_ERR_LINALG, "overlap matrix has fewer independent functions than occupied orbitals");
    std::vector<double> hx(size_t(nb) * m);
    for (int k = 0; k < nb; ++k)   // cuSOLVER's eigenvectors are the columns of a column-major array
      for (int c = 0; c < m; ++c) hx[size_t(k) * m + c] = hv[size_t(keep[c]) * nb + k] / std::sqrt(hs[keep[c]]);
    TCSCF_CUDA(ctx, cudaMemcpyAsync(Xc, hx.data(), sizeof(double) * hx.size(), cudaMemcpyHostToDevice, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  // ---- static operands and the zero start (D = 0: the first build gives F = h, E = 0)
  TCSCF_CUDA(ctx, cudaMemsetAsync(C, 0, sizeof(double) * nb * nocc, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemsetAsync(dD, 0, sizeof(double2) * nn, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemsetAsync(W, 0, sizeof(double) * nb, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemsetAsync(Ws, 0, sizeof(double) * nb, ctx->stream));
  ScfGraphState st0{std::numeric_limits<double>::max(), 0.0, 0, 0, TCSCF_OK, 0};
  TCSCF_CUDA(ctx, cudaMemcpyAsync(st, &st0, sizeof(st0), cudaMemcpyHostToDevice, ctx->stream));
  kWeightedBasis<<<gridBlocks(n2 * nb, 256), 256, 0, ctx->stream>>>(n2, nb, g2.phiR, g2.w, scale, Vw);
  TCSCF_LAUNCH(ctx);
  bool const tensor = precision != TCSCF_PREC_FP64;
  // one grid on both sides: psi1 = psi2 (both C on the same points), the symmetric split-BF16 or FP64
  // contraction (pairs on and above each r1 tile's diagonal; the exchange plus its transpose)
  bool const sym = precision != TCSCF_PREC_TF32 && &g1 == &g2;
  Contraction c;
  c.n1 = n1; c.n2 = n2; c.R = nocc; c.ncol = nb;
  c.p1 = g1.pts; c.p2 = g2.pts; c.psi1 = psi1; c.psi2 = sym ? psi1 : psi2; c.ldpsi = ldpsi;
  c.V = Vw; c.ldv = nb; c.T = Tb; c.ldt = nb; c.coul = coul; c.VH = VH;
  c.sym = sym ? 1 : 0;
  double * FRhalf = nullptr;
  if (sym) TCSCF_TRY(scratch(ctx, "scf_graph_sym_half", sizeof(double) * nn, reinterpret_cast<void **>(&FRhalf)));
  TensorPrep tp;
  TensorPlan plan;
  void * arena = nullptr;
  size_t arenaBytes = 0;
  if (tensor) {
    TCSCF_TRY(tensorPackedV(ctx, g2, Vw, scale, &c.vtPacked));
    TCSCF_TRY(nearPairsFor(ctx, g1, g2, &c.near));
    std::string why;
    TCSCF_CHECK(ctx, tensorPathAvailable(c, precision, &why), TCSCF_ERR_UNSUPPORTED, "graph SCF tensor path: " + why);
    arenaBytes = tensorArenaBytes(c, precision);
    TCSCF_TRY(scratch(ctx, "scf_graph_tensor", arenaBytes, &arena));
    TCSCF_TRY(tensorPrepare(ctx, c, precision, arena, arenaBytes, tp));
    TCSCF_TRY(tensorPlanUpload(ctx, tp, "scf_graph_plan", plan));
  }
  size_t const jacobiSmem = sizeof(double) * size_t(m + (m & 1)) * (m + (m & 1));
  TCSCF_CUDA(ctx, cudaFuncSetAttribute(kJacobiSym, cudaFuncAttributeMaxDynamicSharedMemorySize, int(jacobiSmem)));

  // zeroDensity: the first iteration's density is zero, so its exchange and Coulomb potentials are
  // zero without a contraction (as tcscf_scf skips a rank-0 factor)
  auto body = [&](cudaGraphConditionalHandle handle, int useHandle, bool zeroDensity) -> int {
    if (zeroDensity) {
      TCSCF_CUDA(ctx, cudaMemsetAsync(Tb, 0, sizeof(double) * size_t(n1) * nb, ctx->stream));
      TCSCF_CUDA(ctx, cudaMemsetAsync(VH, 0, sizeof(double) * size_t(n1), ctx->stream));
    } else {
    OrbitalArgs o{n2, nb, nocc, nocc, ldpsi, 0, 0, scale, g2.phiR, g2.w, C, nullptr, sym ? psi1 : psi2, coul, nullptr};
    TCSCF_TRY(orbitals(ctx, o));
    if (!sym) {
      o.n = n1; o.phi = g1.phiR; o.w = g1.w; o.psi = psi1; o.coul = nullptr;
      TCSCF_TRY(orbitals(ctx, o));
    }
    if (tensor) {
      TCSCF_TRY(tensorPrepare(ctx, c, precision, arena, arenaBytes, tp));
      TCSCF_TRY(tensorPlanLaunch(ctx, plan));
      TCSCF_TRY(nearCorrect(ctx, c));
    } else {
      TCSCF_TRY(contractFp64(ctx, c));
    }
    }
    // The exchange of T' and of the skipped pairs in sums of their own.  A split-BF16 build's energies carry a few 1e-8 Eh of
    // rounding, so at which iteration such a loop passes a stop test of that size is chance: any order of these sums moves it, none is
    // better.  Stop test 1e-8 Eh, at most 60 iterations: over 60 Ne grids 12.0 on average in this order, 12.5 as M + M^T (the
    // single builds' form); over 40 Kr grids 43.9 (16 did not pass) and 47.1 (18)
    double const cJ[2] = {2.0, 0.0}, none[2] = {0.0, 0.0};
    TCSCF_TRY(reduceFockReal(ctx, n1, nb, 1, g1.phiR, g1.w, VH, cJ, Tb, 0, nb, FR));
    if (sym) TCSCF_TRY(reduceFockReal(ctx, n1, nb, 1, g1.phiR, g1.w, nullptr, none, Tb, 0, nb, FRhalf));
    TCSCF_TRY(fockFinish(ctx, 1, nb, {FR, nullptr, g1.dsto, sym ? 1 : 0, FRhalf}, dH, dG, nullptr, dD, respectSym, 2.0, dF, dE));
    kScfCheck<<<1, 256, 0, ctx->stream>>>(st, dE, tensor ? plan.status : nullptr, maxIter, tol, int(nn), dD, Dres, nb, Ws, Wres, handle,
                                          useHandle);
    TCSCF_LAUNCH(ctx);
    // the next density from this Fock matrix (real in the real-harmonic basis)
    kDensityToReal<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, g1.dsto, dF, FRc);
    TCSCF_LAUNCH(ctx);
    kSplitDensity<<<1, 256, 0, ctx->stream>>>(nb, FRc, FR, fmaxv);
    TCSCF_LAUNCH(ctx);
    kSmallGemm<<<gridBlocks(int64_t(nb) * m, 256), 256, 0, ctx->stream>>>(nb, m, nb, FR, nb, 0, Xc, m, Tm, m);
    TCSCF_LAUNCH(ctx);
    kSmallGemm<<<gridBlocks(int64_t(m) * m, 256), 256, 0, ctx->stream>>>(m, m, nb, Xc, m, 1, Tm, m, Fp, m);
    TCSCF_LAUNCH(ctx);
    kJacobiSym<<<1, kJacobiThreads, jacobiSmem, ctx->stream>>>(m, Fp, W, Vm);
    TCSCF_LAUNCH(ctx);
    kOccupiedOrbitals<<<1, 256, 0, ctx->stream>>>(nb, m, nocc, W, Vm, Xc, Ws, C, DR);
    TCSCF_LAUNCH(ctx);
    kRealToReference<<<gridBlocks(int64_t(nn), 256), 256, 0, ctx->stream>>>(1, nb, g1.dsto, DR, nullptr, dD);
    TCSCF_LAUNCH(ctx);
    return TCSCF_OK;
  };

  ScfGraphState hst{};
  // the first two iterations directly: the zero-density one, then one that allocates every scratch
  // buffer the body uses
  for (int it = 0; it < 2 && it < maxIter && !hst.done; ++it) {
    TCSCF_TRY(body(0, 0, it == 0));
    TCSCF_CUDA(ctx, cudaMemcpyAsync(&hst, st, sizeof(hst), cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  *graphLaunches = 0;
  if (!hst.done) {
    if (capture) {
      cudaGraph_t graph = nullptr;
      TCSCF_CUDA(ctx, cudaGraphCreate(&graph, 0));
      cudaGraphConditionalHandle handle;
      cudaGraphNode_t node;
      cudaGraphNodeParams cp = {};
      cudaError_t e = cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault);
      if (e == cudaSuccess) {
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = handle;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        e = cudaGraphAddNode(&node, graph, nullptr, 0, &cp);
      }
      if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return fail(ctx, TCSCF_ERR_CUDA, std::string("conditional graph node: ") + cudaGetErrorString(e));
      }
      cudaGraph_t bodyGraph = cp.conditional.phGraph_out[0];
      e = cudaStreamBeginCaptureToGraph(ctx->stream, bodyGraph, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed);
      if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return fail(ctx, TCSCF_ERR_CUDA, std::string("begin capture: ") + cudaGetErrorString(e));
      }
      ctx->capturing = 1;
      int const bst = body(handle, 1, false);
      ctx->capturing = 0;
      cudaGraph_t captured = nullptr;
      e = cudaStreamEndCapture(ctx->stream, &captured);
      if (bst != TCSCF_OK || e != cudaSuccess) {
        cudaGraphDestroy(graph);
        if (bst != TCSCF_OK) return bst;
        return fail(ctx, TCSCF_ERR_CUDA, std::string("end capture: ") + cudaGetErrorString(e));
      }
      cudaGraphExec_t exec = nullptr;
      e = cudaGraphInstantiate(&exec, graph, 0);
      cudaGraphDestroy(graph);
      TCSCF_CHECK(ctx, e == cudaSuccess, TCSCF_ERR_CUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
      e = cudaGraphLaunch(exec, ctx->stream);
      cudaError_t const e2 = cudaStreamSynchronize(ctx->stream);
      cudaGraphExecDestroy(exec);
      TCSCF_CHECK(ctx, e == cudaSuccess && e2 == cudaSuccess, TCSCF_ERR_CUDA,
                  std::string("graph launch: ") + cudaGetErrorString(e != cudaSuccess ? e : e2));
      *graphLaunches = 1;
    } else {
      // the same body launched per iteration, with the host reading the loop state after each
      for (int it = 2; it < maxIter && !hst.done; ++it) {
        TCSCF_TRY(body(0, 0, false));
        TCSCF_CUDA(ctx, cudaMemcpyAsync(&hst, st, sizeof(hst), cudaMemcpyDeviceToHost, ctx->stream));
        TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      }
    }
    TCSCF_CUDA(ctx, cudaMemcpyAsync(&hst, st, sizeof(hst), cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  if (iterations) *iterations = hst.iter;
  if (energy) *energy = hst.eres;
  if (density) TCSCF_CUDA(ctx, cudaMemcpy(density, Dres, sizeof(double2) * nn, cudaMemcpyDeviceToHost));
  if (eigenvalues) {
    std::vector<double> hw(nb, std::numeric_limits<double>::quiet_NaN());
    TCSCF_CUDA(ctx, cudaMemcpy(hw.data(), Wres, sizeof(double) * m, cudaMemcpyDeviceToHost));
    std::copy(hw.begin(), hw.end(), eigenvalues);
  }
  if (hst.code == TCSCF_ERR_TIMEOUT) return fail(ctx, TCSCF_ERR_TIMEOUT, "graph SCF: a bounded wait of the tensor kernel expired");
  if (hst.code == TCSCF_ERR_NONFINITE) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite energy");
  if (hst.code == TCSCF_ERR_NOT_CONVERGED || !hst.done)
    return fail(ctx, TCSCF_ERR_NOT_CONVERGED, "SCF did not converge in " + std::to_string(maxIter) + " iterations");
  return TCSCF_OK;
}

}  // namespace
}  // namespace tcscf

using namespace tcscf;

extern "C" {

int tcscf_ctx_create(int device, tcscf_ctx ** out)
{
  if (!out) return TCSCF_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return TCSCF_ERR_NO_DEVICE;
  if (device < 0 || device >= count) return TCSCF_ERR_INVALID_ARGUMENT;
  if (cudaSetDevice(device) != cudaSuccess) return TCSCF_ERR_CUDA;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return TCSCF_ERR_CUDA;
  if (prop.major != 10) return TCSCF_ERR_UNSUPPORTED;  // built for sm_100a only
  tcscf_ctx * ctx = new tcscf_ctx();
  ctx->device = device;
  if (cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking) != cudaSuccess) { delete ctx; return TCSCF_ERR_CUDA; }
  {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    if (cudaMemPoolCreate(&ctx->gridPool, &props) != cudaSuccess) {
      cudaStreamDestroy(ctx->stream);
      delete ctx;
      return TCSCF_ERR_CUDA;
    }
    // memory of destroyed grids and tensors stays in the pool up to this much (a few Kr-sized grids, the tensors of a Be-TC
    // cycle); the rest goes back to the device at the next synchronisation, and what stays when a cudaMalloc in this
    // process, by the context's scratch or by another user of the device, would fail without it
    uint64_t keep = kPoolKeepBytes;
    cudaMemPoolSetAttribute(ctx->gridPool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  for (auto & e : ctx->ev) cudaEventCreate(&e);
  if (cusolverDnCreate(&ctx->solver) != CUSOLVER_STATUS_SUCCESS) {
    ctx->solver = nullptr;
    tcscf_ctx_destroy(ctx);   // releases the stream, the grid pool and the events made so far
    return TCSCF_ERR_CUDA;
  }
  cusolverDnSetStream(ctx->solver, ctx->stream);
  // the fixed array of tcscf_overlap_core_quadrature_static: its address is looked up here, where
  // allocation is allowed anyway (a lazily loaded module may allocate its globals on first use), so
  // the entry point itself never does set-up work
  double2 * fixedScratch = nullptr;
  if (quadStaticScratch(ctx, &fixedScratch) != TCSCF_OK) {
    tcscf_ctx_destroy(ctx);
    return TCSCF_ERR_CUDA;
  }
  *out = ctx;
  return TCSCF_OK;
}

int tcscf_ctx_destroy(tcscf_ctx * ctx)
{
  if (!ctx) return TCSCF_OK;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  for (auto & kv : ctx->grids) gridReleaseAll(ctx, kv.second);
  for (auto & kv : ctx->tensors) tensorRelease(ctx, kv.second);
  cudaStreamSynchronize(ctx->stream);
  if (ctx->gridPool) cudaMemPoolDestroy(ctx->gridPool);
  for (auto & kv : ctx->scratch) cudaFree(kv.second.p);
  for (auto & kv : ctx->nearPairs)
    if (kv.second.d) cudaFree(kv.second.d);
  for (auto & e : ctx->ev) cudaEventDestroy(e);
  for (auto & e : ctx->tuneEv)
    if (e) cudaEventDestroy(e);
  if (ctx->tensorGraph) cudaGraphExecDestroy(ctx->tensorGraph);
  if (ctx->solver) cusolverDnDestroy(ctx->solver);
  if (ctx->blas) cublasDestroy(ctx->blas);
  cudaStreamDestroy(ctx->stream);
  delete ctx;
  return TCSCF_OK;
}

const char * tcscf_last_error(tcscf_ctx * ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int tcscf_batch_graph_stats(tcscf_ctx * ctx, int * captures, int * replays)
{
  if (!ctx || !captures || !replays) return TCSCF_ERR_INVALID_ARGUMENT;
  *captures = ctx->graphCaptures;
  *replays = ctx->graphReplays;
  return TCSCF_OK;
}

int tcscf_set_autotune(tcscf_ctx * ctx, int enable)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  ctx->autotune = enable ? 1 : 0;
  return TCSCF_OK;
}

int tcscf_autotune_stats(tcscf_ctx * ctx, int * shapes, int * batches, int * measurements)
{
  if (!ctx || !shapes || !batches || !measurements) return TCSCF_ERR_INVALID_ARGUMENT;
  *shapes = int(ctx->tunedSplit.size());
  *batches = int(ctx->tunedBatchPolicy.size());
  *measurements = ctx->tuneMeasurements;
  return TCSCF_OK;
}

int tcscf_autotune_split_candidates(int64_t n1, int64_t n2, int sms, int * splits, int capacity, int * count)
{
  if (n1 <= 0 || n2 <= 0 || sms <= 0 || !count || capacity < 0 || (capacity > 0 && !splits)) return TCSCF_ERR_INVALID_ARGUMENT;
  if (n1 > (int64_t(1) << 36) || n2 > (int64_t(1) << 36)) return TCSCF_ERR_INVALID_ARGUMENT;  // tile and block counts stay int
  std::vector<int> const c = splitCandidates(n1, n2, sms);
  int const n = std::min<int>(capacity, int(c.size()));
  for (int i = 0; i < n; ++i) splits[i] = c[i];
  *count = n;
  return TCSCF_OK;
}

int tcscf_selftest_bounded_wait(tcscf_ctx * ctx, double limit_ms)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  TCSCF_CUDA(ctx, cudaSetDevice(ctx->device));
  return boundedWaitSelfTest(ctx, limit_ms);
}

int tcscf_ctx_stream(tcscf_ctx * ctx, void ** stream)
{
  if (!ctx || !stream) return TCSCF_ERR_INVALID_ARGUMENT;
  *stream = ctx->stream;
  return TCSCF_OK;
}

int tcscf_synchronize(tcscf_ctx * ctx)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

int tcscf_last_timing(tcscf_ctx * ctx, double * contraction_ms, double * total_ms, int * launches)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  if (contraction_ms) *contraction_ms = ctx->lastContractionMs;
  if (total_ms) *total_ms = ctx->lastTotalMs;
  if (launches) *launches = ctx->lastLaunches;
  return TCSCF_OK;
}

int tcscf_last_potentials(tcscf_ctx * ctx, double * VH, double * T)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  TCSCF_CHECK(ctx, ctx->lastVH && ctx->lastT, TCSCF_ERR_INVALID_ARGUMENT, "no direct Fock build has run on this context");
  if (VH) TCSCF_CUDA(ctx, cudaMemcpyAsync(VH, ctx->lastVH, sizeof(double) * ctx->lastN1, cudaMemcpyDeviceToHost, ctx->stream));
  if (T) TCSCF_CUDA(ctx, cudaMemcpyAsync(T, ctx->lastT, sizeof(double) * ctx->lastN1 * ctx->lastNb, cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

int tcscf_grid_create(tcscf_ctx * ctx, const double * points, const double * weights, int64_t n, int ndim, int * grid)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  TCSCF_CHECK(ctx, points && weights && grid && n > 0 && (ndim == 2 || ndim == 3), TCSCF_ERR_INVALID_ARGUMENT, "invalid grid arguments");
  cudaSetDevice(ctx->device);
  Grid g;
  g.n = n;
  g.ndim = ndim;
  if (gridAlloc(ctx, &g.pts, sizeof(double) * 3 * n) != TCSCF_OK || gridAlloc(ctx, &g.w, sizeof(double) * n) != TCSCF_OK) {
    std::string const msg = ctx->err;
    gridReleaseAll(ctx, g);
    return fail(ctx, TCSCF_ERR_CUDA, msg);
  }
  if (ndim == 3) TCSCF_CUDA(ctx, cudaMemcpyAsync(g.pts, points, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, ctx->stream));
  else {
    TCSCF_CUDA(ctx, cudaMemcpyAsync(g.pts, points, sizeof(double) * n, cudaMemcpyHostToDevice, ctx->stream));
    TCSCF_CUDA(ctx, cudaMemsetAsync(g.pts + n, 0, sizeof(double) * n, ctx->stream));
    TCSCF_CUDA(ctx, cudaMemcpyAsync(g.pts + 2 * n, points + n, sizeof(double) * n, cudaMemcpyHostToDevice, ctx->stream));
  }
  TCSCF_CUDA(ctx, cudaMemcpyAsync(g.w, weights, sizeof(double) * n, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  int const id = ctx->nextId++;
  ctx->grids[id] = g;
  *grid = id;
  return TCSCF_OK;
}

int tcscf_grid_destroy(tcscf_ctx * ctx, int grid)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  Grid * g = findGrid(ctx, grid);
  TCSCF_CHECK(ctx, g, TCSCF_ERR_INVALID_ARGUMENT, "unknown grid handle");
  nearPairsForget(ctx, g);
  gridReleaseAll(ctx, *g);
  ctx->grids.erase(grid);
  return TCSCF_OK;
}

int tcscf_near_coincident_pairs(tcscf_ctx * ctx, int r1, int r2, int * count)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  TCSCF_CUDA(ctx, cudaSetDevice(ctx->device));
  Grid * g1 = findGrid(ctx, r1);
  Grid * g2 = findGrid(ctx, r2);
  TCSCF_CHECK(ctx, g1 && g2 && count, TCSCF_ERR_INVALID_ARGUMENT, "unknown grid handle or null count");
  NearList const * nl = nullptr;
  TCSCF_TRY(nearPairsFor(ctx, *g1, *g2, &nl));
  *count = nl->count;
  return TCSCF_OK;
}

int tcscf_grid_set_basis(tcscf_ctx * ctx, int grid, const tcscf_sto * basis, int nb, int gradients)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  Grid * g = findGrid(ctx, grid);
  TCSCF_CHECK(ctx, g, TCSCF_ERR_INVALID_ARGUMENT, "unknown grid handle");
  std::vector<DevSto> ds;
  TCSCF_TRY(validateBasis(ctx, basis, nb, ds));
  TCSCF_CHECK(ctx, !(gradients && basis[0].family == TCSCF_BASIS_HYDROGEN), TCSCF_ERR_UNSUPPORTED,
              "hydrogen-like functions have no gradient (HydrogenLikeBasis.hpp:51-55)");
  gridRelease(ctx, g->dsto); gridRelease(ctx, g->phiR); gridRelease(ctx, g->vals); gridRelease(ctx, g->grads);
  gridRelease(ctx, g->vtCache);
  g->dsto = nullptr; g->phiR = g->vals = g->grads = nullptr;
  g->vtCache = nullptr;
  g->vtNB = 0;
  g->nb = 0;
  TCSCF_TRY(gridAlloc(ctx, &g->dsto, sizeof(DevSto) * nb));
  TCSCF_TRY(gridAlloc(ctx, &g->phiR, sizeof(double) * g->n * nb));
  TCSCF_TRY(gridAlloc(ctx, &g->vals, sizeof(double) * g->n * nb * (g->ndim == 3 ? 2 : 1)));
  if (gradients) TCSCF_TRY(gridAlloc(ctx, &g->grads, sizeof(double) * g->n * nb * 6));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(g->dsto, ds.data(), sizeof(DevSto) * nb, cudaMemcpyHostToDevice, ctx->stream));
  int lmax = 0;
  for (DevSto const & d : ds) lmax = std::max(lmax, d.l);
  // about four (point, function) pairs a thread (a point a thread at most: the tables' chains of functions are theirs), fewer where the
  // points are few (two blocks per SM), the tables within 48 KB (8 points of lmax = 12 take 8.4 KB).
  // At least 8 and at most 64 points whatever their number: 34 us a call for 27 here at 50 points x 12 functions, 36 for 28 at 20, 40 for 30 at 400,000 x 1
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  int const share = int(std::min<int64_t>(256, (g->n + 2 * sms - 1) / (2 * sms)));
  int const npts = std::min({std::max(8, std::min(256, 1024 / nb)), std::max(1, share), int(48 * 1024 / (sizeof(double) * basisPointDoubles(lmax)))});
  kBasis<<<unsigned((g->n + npts - 1) / npts), 256, sizeof(double) * npts * basisPointDoubles(lmax), ctx->stream>>>(
    g->n, nb, g->ndim, lmax, npts, g->pts, g->dsto, g->phiR, g->vals, g->grads);
  TCSCF_LAUNCH(ctx);
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  g->nb = nb;
  g->hasGrad = gradients ? 1 : 0;
  g->basis.assign(basis, basis + nb);
  return TCSCF_OK;
}

int tcscf_grid_basis_values(tcscf_ctx * ctx, int grid, double * values, double * gradients)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  Grid * g = findGrid(ctx, grid);
  TCSCF_CHECK(ctx, g && g->nb > 0, TCSCF_ERR_INVALID_ARGUMENT, "grid has no basis");
  if (values)
    TCSCF_CUDA(ctx, cudaMemcpyAsync(values, g->vals, sizeof(double) * g->n * g->nb * (g->ndim == 3 ? 2 : 1), cudaMemcpyDeviceToHost, ctx->stream));
  if (gradients) {
    TCSCF_CHECK(ctx, g->grads, TCSCF_ERR_INVALID_ARGUMENT, "gradients were not stored");
    TCSCF_CUDA(ctx, cudaMemcpyAsync(gradients, g->grads, sizeof(double) * g->n * g->nb * 6, cudaMemcpyDeviceToHost, ctx->stream));
  }
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

int tcscf_overlap_core_quadrature(tcscf_ctx * ctx, int grid, int Z, double * S, double * H)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  Grid * g = findGrid(ctx, grid);
  TCSCF_CHECK(ctx, g && g->nb > 0 && g->ndim == 3, TCSCF_ERR_INVALID_ARGUMENT, "needs a 3-D grid with a basis");
  TCSCF_CHECK(ctx, S, TCSCF_ERR_INVALID_ARGUMENT, "S is required");
  TCSCF_CHECK(ctx, !H || g->grads, TCSCF_ERR_INVALID_ARGUMENT, "H needs stored gradients");
  int const nb = g->nb;
  void * p = nullptr;
  int const chunks = quadChunks(ctx, *g);
  TCSCF_TRY(scratch(ctx, "quad_sh", sizeof(double2) * nb * nb * 2 * (size_t(chunks) + 1), &p));
  double2 * dS = static_cast<double2 *>(p);
  double2 * dH = dS + nb * nb;
  TCSCF_TRY(quadLaunch(ctx, *g, Z, H != nullptr, dS, chunks));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(S, dS, sizeof(double2) * nb * nb, cudaMemcpyDeviceToHost, ctx->stream));
  if (H) TCSCF_CUDA(ctx, cudaMemcpyAsync(H, dH, sizeof(double2) * nb * nb, cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

// Fixed-scratch form of the S/H quadrature: results and partial sums go to a file-scope device array
// instead of context scratch, so this entry point allocates nothing.  It serves callers that cannot
// allocate device memory at this point: a host whose device memory is already handed out to its own
// pool (grids and tensors sized to fill HBM), and a host that cannot accept the device-wide
// synchronisation that cudaFree implies while its other streams are running.
//   * Limit: nb <= kQuadStaticMaxNb (256), i.e. 2 x 256 x 256 complex doubles = 2 MiB per device;
//     larger bases are rejected with TCSCF_ERR_UNSUPPORTED.
//   * Set-up: tcscf_ctx_create looks up the array's device address (cudaGetSymbolAddress, with the
//     context's device current), so a call of this entry point does no set-up of its own.
//   * Sharing: every call on a device uses the same array, so overlapping calls on one device (other
//     streams or other contexts) race; callers serialise them.  Nothing in the array needs to start
//     at zero: every element is written before it is read.
int tcscf_overlap_core_quadrature_static(tcscf_ctx * ctx, int grid, int Z, double * S, double * H)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  Grid * g = findGrid(ctx, grid);
  TCSCF_CHECK(ctx, g && g->nb > 0 && g->ndim == 3, TCSCF_ERR_INVALID_ARGUMENT, "needs a 3-D grid with a basis");
  TCSCF_CHECK(ctx, S, TCSCF_ERR_INVALID_ARGUMENT, "S is required");
  TCSCF_CHECK(ctx, !H || g->grads, TCSCF_ERR_INVALID_ARGUMENT, "H needs stored gradients");
  int const nb = g->nb;
  TCSCF_CHECK(ctx, nb <= kQuadStaticMaxNb, TCSCF_ERR_UNSUPPORTED,
              "nb = " + std::to_string(nb) + " exceeds the fixed scratch of tcscf_overlap_core_quadrature_static (nb <= " +
                  std::to_string(kQuadStaticMaxNb) + "); use tcscf_overlap_core_quadrature");
  TCSCF_CUDA(ctx, cudaSetDevice(ctx->device));
  double2 * dS = nullptr;
  TCSCF_TRY(quadStaticScratch(ctx, &dS));
  double2 * dH = dS + nb * nb;
  // as many chunks of partial sums as the array holds behind S and H (none at nb = 256)
  int const room = (kQuadStaticMaxNb * kQuadStaticMaxNb) / (nb * nb) - 1;
  TCSCF_TRY(quadLaunch(ctx, *g, Z, H != nullptr, dS, std::max(1, room)));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(S, dS, sizeof(double2) * nb * nb, cudaMemcpyDeviceToHost, ctx->stream));
  if (H) TCSCF_CUDA(ctx, cudaMemcpyAsync(H, dH, sizeof(double2) * nb * nb, cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

int tcscf_fock_build(tcscf_ctx * ctx, int r1, int r2, int nspin, const double * density, const double * h, int respect_symmetry,
                     int precision, double * G, double * fock, double * energy)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  Grid * g1 = findGrid(ctx, r1);
  Grid * g2 = findGrid(ctx, r2);
  TCSCF_TRY(checkBasisPair(ctx, g1, g2));
  TCSCF_CHECK(ctx, nspin == 1 || nspin == 2, TCSCF_ERR_INVALID_ARGUMENT, "nspin must be 1 or 2");
  TCSCF_CHECK(ctx, density && h, TCSCF_ERR_INVALID_ARGUMENT, "density and h are required");
  TCSCF_CHECK(ctx, precision >= TCSCF_PREC_FP64 && precision <= TCSCF_PREC_TF32, TCSCF_ERR_INVALID_ARGUMENT, "unknown precision");
  int const nb = g1->nb;
  size_t const nn = size_t(nb) * nb;
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "fock_io", sizeof(double2) * nn * nspin * 3 + sizeof(double) * nn + 64, &p));
  double2 * dD = static_cast<double2 *>(p);
  double2 * dG = dD + nn * nspin;
  double2 * dF = dG + nn * nspin;
  double * dH = reinterpret_cast<double *>(dF + nn * nspin);
  double * dE = dH + nn;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dD, density, sizeof(double2) * nn * nspin, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dH, h, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_TRY(fockBuildDevice(ctx, *g1, *g2, nspin, dD, dH, respect_symmetry, precision, dG, dF, dE, nullptr));
  if (G) TCSCF_CUDA(ctx, cudaMemcpyAsync(G, dG, sizeof(double2) * nn * nspin, cudaMemcpyDeviceToHost, ctx->stream));
  if (fock) TCSCF_CUDA(ctx, cudaMemcpyAsync(fock, dF, sizeof(double2) * nn * nspin, cudaMemcpyDeviceToHost, ctx->stream));
  double e = 0;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(&e, dE, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (energy) *energy = e;
  if (!(e == e) || std::isinf(e)) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite energy");
  return TCSCF_OK;
}

int tcscf_fock_build_device(tcscf_ctx * ctx, int r1, int r2, int nspin, const double * density, const double * h, int respect_symmetry,
                            int precision, double * G, double * fock, double * energy)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  Grid * g1 = findGrid(ctx, r1);
  Grid * g2 = findGrid(ctx, r2);
  TCSCF_TRY(checkBasisPair(ctx, g1, g2));
  TCSCF_CHECK(ctx, nspin == 1 || nspin == 2, TCSCF_ERR_INVALID_ARGUMENT, "nspin must be 1 or 2");
  TCSCF_CHECK(ctx, density && h && energy, TCSCF_ERR_INVALID_ARGUMENT, "density, h and energy are required");
  TCSCF_CHECK(ctx, precision >= TCSCF_PREC_FP64 && precision <= TCSCF_PREC_TF32, TCSCF_ERR_INVALID_ARGUMENT, "unknown precision");
  size_t const nn = size_t(g1->nb) * g1->nb;
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "fock_dev_io", sizeof(double2) * nn * nspin * 2, &p));
  double2 * dG = G ? reinterpret_cast<double2 *>(G) : static_cast<double2 *>(p);
  double2 * dF = fock ? reinterpret_cast<double2 *>(fock) : static_cast<double2 *>(p) + nn * nspin;
  TCSCF_TRY(fockBuildDevice(ctx, *g1, *g2, nspin, reinterpret_cast<const double2 *>(density), h, respect_symmetry, precision, dG, dF, energy,
                            nullptr));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return TCSCF_OK;
}

int tcscf_compute_F(tcscf_ctx * ctx, int r1, int r2, int kernel, const tcscf_ochi * jastrow, int precision, double * F, int keep,
                    int * fji)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  TCSCF_CHECK(ctx, kernel >= TCSCF_K_INV_R12 && kernel <= TCSCF_K_TC_SCALAR_OPPO, TCSCF_ERR_INVALID_ARGUMENT, "computeF takes a scalar kernel");
  TCSCF_CHECK(ctx, kernel == TCSCF_K_INV_R12 || jastrow, TCSCF_ERR_INVALID_ARGUMENT, "TC kernels need the Jastrow parameters");
  return precomputeTensor(ctx, r1, r2, kernel, jastrow, precision, 1, F, keep, fji);
}

int tcscf_compute_V(tcscf_ctx * ctx, int r1, int r2, int kernel, const tcscf_ochi * jastrow, int precision, double * V, int keep,
                    int * vji)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  TCSCF_CHECK(ctx, kernel == TCSCF_K_GRAD_U_SAME || kernel == TCSCF_K_GRAD_U_OPPO, TCSCF_ERR_INVALID_ARGUMENT, "computeV takes a vector kernel");
  TCSCF_CHECK(ctx, jastrow, TCSCF_ERR_INVALID_ARGUMENT, "Jastrow parameters required");
  return precomputeTensor(ctx, r1, r2, kernel, jastrow, precision, 3, V, keep, vji);
}

int tcscf_tensor_destroy(tcscf_ctx * ctx, int handle)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  auto it = ctx->tensors.find(handle);
  TCSCF_CHECK(ctx, it != ctx->tensors.end(), TCSCF_ERR_INVALID_ARGUMENT, "unknown tensor handle");
  tensorRelease(ctx, it->second);
  ctx->tensors.erase(it);
  // the pool gives memory back when the stream is synchronised: here where it holds more unused memory than it is to keep, so that
  // the rest is the device's again when this returns (always: 4 us of a 47 us computeF and destroy, and memory that the next tensors
  // would take again goes to the device and back)
  uint64_t held = 0, used = 0;
  cudaMemPoolGetAttribute(ctx->gridPool, cudaMemPoolAttrReservedMemCurrent, &held);
  cudaMemPoolGetAttribute(ctx->gridPool, cudaMemPoolAttrUsedMemCurrent, &used);
  if (held - used > kPoolKeepBytes) cudaStreamSynchronize(ctx->stream);
  return TCSCF_OK;
}

int tcscf_fock_build_batch(tcscf_ctx * ctx, int count, const int * r1, const int * r2, const double * const * density,
                           const double * const * h, int respect_symmetry, int precision, double * energy, double * const * fock)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  TCSCF_CHECK(ctx, count >= 1 && r1 && r2 && density && h && energy, TCSCF_ERR_INVALID_ARGUMENT, "batch: count, grids, densities, h and energy are required");
  TCSCF_CHECK(ctx, precision >= TCSCF_PREC_FP64 && precision <= TCSCF_PREC_TF32, TCSCF_ERR_INVALID_ARGUMENT, "unknown precision");
  std::vector<Grid *> g1s(count), g2s(count);
  size_t io = 0;
  for (int k = 0; k < count; ++k) {
    g1s[k] = findGrid(ctx, r1[k]);
    g2s[k] = findGrid(ctx, r2[k]);
    TCSCF_TRY(checkBasisPair(ctx, g1s[k], g2s[k]));
    TCSCF_CHECK(ctx, density[k] && h[k], TCSCF_ERR_INVALID_ARGUMENT, "batch: every instance needs a density and h");
    size_t const nn = size_t(g1s[k]->nb) * g1s[k]->nb;
    io += sizeof(double2) * 3 * nn + sizeof(double) * nn + 256;
  }
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "batch_io", io + sizeof(double) * count + 256, &p));
  std::vector<const double2 *> dD(count);
  std::vector<const double *> dH(count);
  std::vector<double2 *> dG(count), dF(count);
  std::vector<double *> dE(count);
  char * q = static_cast<char *>(p);
  double * energies = reinterpret_cast<double *>(q);
  q += (sizeof(double) * count + 255) & ~size_t(255);
  for (int k = 0; k < count; ++k) {
    size_t const nn = size_t(g1s[k]->nb) * g1s[k]->nb;
    auto * d = reinterpret_cast<double2 *>(q);
    dD[k] = d; dG[k] = d + nn; dF[k] = d + 2 * nn;
    auto * hh = reinterpret_cast<double *>(d + 3 * nn);
    dH[k] = hh;
    dE[k] = energies + k;
    q += (sizeof(double2) * 3 * nn + sizeof(double) * nn + 255) & ~size_t(255);
    TCSCF_CUDA(ctx, cudaMemcpyAsync(d, density[k], sizeof(double2) * nn, cudaMemcpyHostToDevice, ctx->stream));
    TCSCF_CUDA(ctx, cudaMemcpyAsync(hh, h[k], sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  }
  auto build = [&]() {
    return fockBuildBatch(ctx, count, g1s.data(), g2s.data(), dD.data(), dH.data(), respect_symmetry, precision, dG.data(), dF.data(), dE.data());
  };
  if (ctx->autotune && (precision == TCSCF_PREC_BF16X3 || precision == TCSCF_PREC_TF32)) {
    // batch signature: precision and every instance's grid sizes and basis size
    std::vector<int64_t> key{precision, count};
    for (int k = 0; k < count; ++k) key.insert(key.end(), {g1s[k]->n, g2s[k]->n, int64_t(g1s[k]->nb)});
    auto it = ctx->tunedBatchPolicy.find(key);
    if (it == ctx->tunedBatchPolicy.end()) {
      // each policy's whole batch build runs twice and the second (its graph replayed, scratch
      // grown) is timed between the build's own events; the inputs are read-only, so every run
      // writes the same outputs up to the order of the r2 sums
      int best = 1;
      double bestMs = 0;
      bool first = true;
      for (int policy : {1, 0, 2, 4}) {
        ctx->batchSplitPolicy = policy;
        int st = build();
        if (st == TCSCF_OK) st = build();
        if (st != TCSCF_OK) { ctx->batchSplitPolicy = 1; return st; }
        ++ctx->tuneMeasurements;
        if (first || ctx->lastTotalMs < bestMs) { bestMs = ctx->lastTotalMs; best = policy; }
        first = false;
      }
      it = ctx->tunedBatchPolicy.emplace(key, best).first;
    }
    ctx->batchSplitPolicy = it->second;
  }
  int const bst = build();
  ctx->batchSplitPolicy = 1;
  TCSCF_TRY(bst);
  TCSCF_CUDA(ctx, cudaMemcpyAsync(energy, energies, sizeof(double) * count, cudaMemcpyDeviceToHost, ctx->stream));
  for (int k = 0; k < count; ++k)
    if (fock && fock[k])
      TCSCF_CUDA(ctx, cudaMemcpyAsync(fock[k], dF[k], sizeof(double2) * g1s[k]->nb * g1s[k]->nb, cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int k = 0; k < count; ++k)
    if (!(energy[k] == energy[k]) || std::isinf(energy[k])) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite energy in batch instance " + std::to_string(k));
  return TCSCF_OK;
}

int tcscf_fock_build_precomputed(tcscf_ctx * ctx, int r1, int fji, int nspin, const double * density, const double * h,
                                 int respect_symmetry, double * G, double * fock, double * energy)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  Grid * g1 = findGrid(ctx, r1);
  TCSCF_CHECK(ctx, g1 && g1->nb > 0 && g1->ndim == 3, TCSCF_ERR_INVALID_ARGUMENT, "r1 grid needs a basis");
  auto it = ctx->tensors.find(fji);
  TCSCF_CHECK(ctx, it != ctx->tensors.end() && !it->second.vec, TCSCF_ERR_INVALID_ARGUMENT, "unknown Fji handle");
  Tensor const & t = it->second;
  TCSCF_CHECK(ctx, t.n1 == g1->n && t.nb == g1->nb, TCSCF_ERR_INVALID_ARGUMENT, "Fji does not match the r1 grid");
  TCSCF_CHECK(ctx, nspin == 1 || nspin == 2, TCSCF_ERR_INVALID_ARGUMENT, "nspin must be 1 or 2");
  TCSCF_CHECK(ctx, density && h, TCSCF_ERR_INVALID_ARGUMENT, "density and h are required");
  int const nb = g1->nb;
  int64_t const n1 = g1->n;
  size_t const nn = size_t(nb) * nb;
  void * p = nullptr;
  TCSCF_CHECK(ctx, nb <= kFaiMaxNb, TCSCF_ERR_UNSUPPORTED, "precompute-form Fock reduction supports nb <= 64");
  size_t const fai = size_t(nspin) * n1 * nb;
  TCSCF_TRY(scratch(ctx, "fock_pre", sizeof(double2) * nn * nspin * 4 + sizeof(double) * (2 * fai + 2 * n1 + 2 * nn * nspin + nn + 8), &p));
  double2 * dD = static_cast<double2 *>(p);
  double2 * dG = dD + nn * nspin;
  double2 * dF = dG + nn * nspin;
  double2 * DR = dF + nn * nspin;
  double * FaiRe = reinterpret_cast<double *>(DR + nn * nspin);
  double * FaiIm = FaiRe + fai;
  double * FaaRe = FaiIm + fai;
  double * FaaIm = FaaRe + n1;
  double * GRre = FaaIm + n1;
  double * GRim = GRre + nn * nspin;
  double * dH = GRim + nn * nspin;
  double * dE = dH + nn;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dD, density, sizeof(double2) * nn * nspin, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dH, h, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  cudaEventRecord(ctx->ev[0], ctx->stream);
  int const launch0 = ctx->launchCount;
  for (int s = 0; s < nspin; ++s) TCSCF_TRY(densityToRealLaunch(ctx, nb, g1->dsto, dD + s * nn, DR + s * nn));
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  size_t const sm = sizeof(double2) * nn * nspin;
  auto launch = [&](auto kernel) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm));
    int per = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 256, sm);
    kernel<<<unsigned(std::min<int64_t>(n1, int64_t(sms) * std::max(per, 1))), 256, sm, ctx->stream>>>(n1, nb, tensorStride(nb), tensorPlane(nb), t.d, g1->phiR, DR, FaaRe, FaaIm, FaiRe, FaiIm);
  };
  if (nspin == 1) launch(kFaaFai<1>);
  else launch(kFaaFai<2>);
  TCSCF_LAUNCH(ctx);
  // G = sum_r w phi (cJ phi Faa - Fai), real and imaginary parts apart
  double const cJ0 = nspin == 1 ? 2.0 : 1.0, cJ[2] = {cJ0, cJ0};
  TCSCF_TRY(reduceFockReal(ctx, n1, nb, nspin, g1->phiR, g1->w, FaaRe, cJ, FaiRe, int64_t(n1) * nb, nb, GRre));
  TCSCF_TRY(reduceFockReal(ctx, n1, nb, nspin, g1->phiR, g1->w, FaaIm, cJ, FaiIm, int64_t(n1) * nb, nb, GRim));
  TCSCF_TRY(fockFinish(ctx, nspin, nb, {GRre, GRim, g1->dsto, 0}, dH, dG, nullptr, dD, respect_symmetry, cJ0, dF, dE));
  cudaEventRecord(ctx->ev[1], ctx->stream);
  if (G) TCSCF_CUDA(ctx, cudaMemcpyAsync(G, dG, sizeof(double2) * nn * nspin, cudaMemcpyDeviceToHost, ctx->stream));
  if (fock) TCSCF_CUDA(ctx, cudaMemcpyAsync(fock, dF, sizeof(double2) * nn * nspin, cudaMemcpyDeviceToHost, ctx->stream));
  double e = 0;
  TCSCF_CUDA(ctx, cudaMemcpyAsync(&e, dE, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  float ms = 0;
  cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
  ctx->lastTotalMs = ms;
  ctx->lastContractionMs = ms;
  ctx->lastLaunches = ctx->launchCount - launch0;
  if (energy) *energy = e;
  if (!(e == e) || std::isinf(e)) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite energy");
  return TCSCF_OK;
}

int tcscf_set_scf_options(tcscf_ctx * ctx, int diis, int real_eigensolve)
{
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  TCSCF_CHECK(ctx, diis >= 0 && diis <= 16, TCSCF_ERR_INVALID_ARGUMENT, "DIIS history must be 0..16");
  ctx->diisSize = diis == 1 ? 0 : diis;
  ctx->realEigen = real_eigensolve ? 1 : 0;
  return TCSCF_OK;
}

int tcscf_scf(tcscf_ctx * ctx, int r1, int r2, int nspin, int n_up, int n_down, const double * S, const double * h, int respect_symmetry,
              int precision, double tol, int max_iter, double * energy, int * iterations, double * density, double * eigenvalues)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  Grid * g1 = findGrid(ctx, r1);
  Grid * g2 = findGrid(ctx, r2);
  TCSCF_TRY(checkBasisPair(ctx, g1, g2));
  TCSCF_CHECK(ctx, nspin == 1 || nspin == 2, TCSCF_ERR_INVALID_ARGUMENT, "nspin must be 1 or 2");
  TCSCF_CHECK(ctx, S && h && max_iter > 0, TCSCF_ERR_INVALID_ARGUMENT, "S, h and max_iter are required");
  // RCSHartreeFock requires an even electron count (HartreeFock.hpp:248)
  TCSCF_CHECK(ctx, nspin == 2 || (n_up + n_down) % 2 == 0, TCSCF_ERR_INVALID_ARGUMENT, "RCS needs an even electron count");
  int const nb = g1->nb;
  int const nocc[2] = {nspin == 1 ? (n_up + n_down) / 2 : n_up, n_down};
  TCSCF_CHECK(ctx, nocc[0] <= nb && nocc[1] <= nb && nocc[0] >= 0 && nocc[1] >= 0, TCSCF_ERR_INVALID_ARGUMENT, "more electrons than basis functions");
  size_t const nn = size_t(nb) * nb;
  void * p = nullptr;
  TCSCF_TRY(scratch(ctx, "scf", sizeof(double2) * (nn * nspin * 3 + nn * 2) + sizeof(double) * (nn * 2 + nb * nspin + 16), &p));
  double2 * dD = static_cast<double2 *>(p);
  double2 * dG = dD + nn * nspin;
  double2 * dF = dG + nn * nspin;
  double2 * A = dF + nn * nspin;
  double2 * B = A + nn;
  double * dH = reinterpret_cast<double *>(B + nn);
  double * dS = dH + nn;
  double * W = dS + nn;
  double * dE = W + nb * nspin;
  int * devInfo = reinterpret_cast<int *>(dE + 8);
  TCSCF_CUDA(ctx, cudaMemsetAsync(dD, 0, sizeof(double2) * nn * nspin, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dH, h, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  TCSCF_CUDA(ctx, cudaMemcpyAsync(dS, S, sizeof(double) * nn, cudaMemcpyHostToDevice, ctx->stream));
  int lwork = 0;
  if (cusolverDnZhegvd_bufferSize(ctx->solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, nb,
                                  reinterpret_cast<cuDoubleComplex *>(A), nb, reinterpret_cast<cuDoubleComplex *>(B), nb, W, &lwork) != CUSOLVER_STATUS_SUCCESS)
    return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnZhegvd_bufferSize failed");
  void * wk = nullptr;
  TCSCF_TRY(scratch(ctx, "hegvd_work", sizeof(double2) * size_t(lwork) + 64, &wk));
  // optional Pulay DIIS: history of Fock matrices and commutator errors FDS - SDF (both spins)
  int const nd = ctx->diisSize;
  size_t const len = size_t(nspin) * nn;
  double2 * Fh = nullptr, * Eh = nullptr, * T1 = nullptr, * T2 = nullptr, * Sc = nullptr, * Fd = nullptr;
  double * dDots = nullptr, * dCoef = nullptr;
  cublasHandle_t bh = nullptr;
  std::vector<double> Bm(size_t(nd) * nd, 0.0), hDots(nd), coef;
  int count = 0, head = 0;
  {
    void * q = nullptr;
    TCSCF_TRY(scratch(ctx, "scf_diis", sizeof(double2) * (2 * size_t(nd) * len + 3 * nn + len) + sizeof(double) * 2 * (nd + 1) + 1024, &q));
    Fh = static_cast<double2 *>(q);
    Eh = Fh + size_t(nd) * len;
    T1 = Eh + size_t(nd) * len;
    T2 = T1 + nn;
    Sc = T2 + nn;
    Fd = Sc + nn;
    dDots = reinterpret_cast<double *>(Fd + len);
    dCoef = dDots + nd + 1;
    kRealToComplex<<<gridBlocks(int64_t(nn), 256), 256, 0, ctx->stream>>>(int64_t(nn), dS, Sc);
    TCSCF_LAUNCH(ctx);
    if (nd > 0) TCSCF_TRY(blasHandle(ctx, &bh));
  }
  // Optional real-harmonic eigen-solve (tcscf_set_scf_options): the Fock matrix of a density that is
  // real in the real-harmonic basis is real there too, and the real symmetric problem
  // (cusolverDnDsygvd) gives real eigenvectors, so the next density stays real (one rank-nocc tensor
  // contraction per build) even when the aufbau occupation splits a degenerate shell, where the complex
  // solver of the reference basis returns arbitrary complex combinations (doubling the factor rank
  // and the contractions).  Same eigenvalues; when a degenerate level is partly occupied the two
  // solvers occupy different members of it, so the default keeps the reference's complex path.
  void * rp = nullptr;
  TCSCF_TRY(scratch(ctx, "scf_real", sizeof(double2) * 2 * nn + sizeof(double) * 5 * nn + 256, &rp));
  double2 * FR = static_cast<double2 *>(rp);
  double2 * SRc = FR + nn;
  double * Ar = reinterpret_cast<double *>(SRc + nn);
  double * Br = Ar + nn;
  double * SRre = Br + nn;
  double * DRre = SRre + nn;
  double * fmax = DRre + nn;
  bool realPath = true;
  int lworkR = 0;
  void * wkR = nullptr;
  {
    kDensityToReal<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, g1->dsto, Sc, SRc);
    TCSCF_LAUNCH(ctx);
    kSplitDensity<<<1, 256, 0, ctx->stream>>>(nb, SRc, SRre, fmax);
    TCSCF_LAUNCH(ctx);
    double hm[2];
    TCSCF_CUDA(ctx, cudaMemcpyAsync(hm, fmax, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    realPath = ctx->realEigen && hm[1] <= 1e-12 * hm[0];
    if (realPath) {
      if (cusolverDnDsygvd_bufferSize(ctx->solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, nb, Ar, nb, Br, nb, W,
                                      &lworkR) != CUSOLVER_STATUS_SUCCESS)
        return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnDsygvd_bufferSize failed");
      TCSCF_TRY(scratch(ctx, "sygvd_work", sizeof(double) * size_t(lworkR) + 64, &wkR));
    }
  }
  double2 const one = make_double2(1, 0), zero = make_double2(0, 0), mone = make_double2(-1, 0);
  double e = std::numeric_limits<double>::max();
  // density factors from the previous iteration's real-harmonic eigen-solve (every spin solved real)
  Factor given[2];
  bool givenOk = false;
  double * Xocc = nullptr;
  if (realPath) TCSCF_TRY(scratch(ctx, "scf_occ_factor", sizeof(double) * 2 * nn + 64, reinterpret_cast<void **>(&Xocc)));
  for (int it = 0; it < max_iter; ++it) {
    TCSCF_TRY(fockBuildDevice(ctx, *g1, *g2, nspin, dD, dH, respect_symmetry, precision, dG, dF, dE, givenOk ? given : nullptr));
    double ne = 0;
    TCSCF_CUDA(ctx, cudaMemcpyAsync(&ne, dE, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (!(ne == ne) || std::isinf(ne)) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite energy");
    if (iterations) *iterations = it + 1;
    if (std::fabs(ne - e) < tol) {
      if (energy) *energy = ne;
      if (density) TCSCF_CUDA(ctx, cudaMemcpy(density, dD, sizeof(double2) * nn * nspin, cudaMemcpyDeviceToHost));
      if (eigenvalues) TCSCF_CUDA(ctx, cudaMemcpy(eigenvalues, W, sizeof(double) * nb * nspin, cudaMemcpyDeviceToHost));
      return TCSCF_OK;
    }
    e = ne;
    const double2 * Fuse = dF;
    if (nd > 0 && it >= 1) {
      int const slot = head;
      head = (head + 1) % nd;
      count = std::min(count + 1, nd);
      for (int s = 0; s < nspin; ++s) {
        double2 const * Fs = dF + s * nn;
        double2 const * Ds = dD + s * nn;
        double2 * Es = Eh + slot * len + s * nn;
        TCSCF_TRY(rowMajorZgemm(ctx, bh, nb, one, Ds, Sc, zero, T1));     // D S
        TCSCF_TRY(rowMajorZgemm(ctx, bh, nb, one, Fs, T1, zero, Es));     // F D S
        TCSCF_TRY(rowMajorZgemm(ctx, bh, nb, one, Sc, Ds, zero, T2));     // S D
        TCSCF_TRY(rowMajorZgemm(ctx, bh, nb, mone, T2, Fs, one, Es));     // - S D F
        TCSCF_CUDA(ctx, cudaMemcpyAsync(Fh + slot * len + s * nn, Fs, sizeof(double2) * nn, cudaMemcpyDeviceToDevice, ctx->stream));
      }
      kDiisDots<<<count, 256, 0, ctx->stream>>>(int64_t(len), slot, count, Eh, dDots);
      TCSCF_LAUNCH(ctx);
      TCSCF_CUDA(ctx, cudaMemcpyAsync(hDots.data(), dDots, sizeof(double) * count, cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      for (int j = 0; j < count; ++j) Bm[slot * nd + j] = Bm[j * nd + slot] = hDots[j];
      if (count >= 2) {
        // equations scaled by the largest error norm for conditioning
        double mx = 0;
        for (int j = 0; j < count; ++j) mx = std::max(mx, Bm[j * nd + j]);
        std::vector<double> Bs(size_t(count) * count);
        for (int i = 0; i < count; ++i)
          for (int j = 0; j < count; ++j) Bs[i * count + j] = mx > 0 ? Bm[i * nd + j] / mx : Bm[i * nd + j];
        if (mx > 0 && solveDiis(count, Bs, count, coef)) {
          TCSCF_CUDA(ctx, cudaMemcpyAsync(dCoef, coef.data(), sizeof(double) * count, cudaMemcpyHostToDevice, ctx->stream));
          kDiisCombine<<<gridBlocks(int64_t(len), 256), 256, 0, ctx->stream>>>(int64_t(len), count, dCoef, Fh, Fd);
          TCSCF_LAUNCH(ctx);
          Fuse = Fd;
        }
      }
    }
    int solvedReal = 0;
    given[0] = given[1] = Factor{};
    for (int s = 0; s < nspin; ++s) {
      if (realPath) {
        kDensityToReal<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, g1->dsto, Fuse + s * nn, FR);
        TCSCF_LAUNCH(ctx);
        kSplitDensity<<<1, 256, 0, ctx->stream>>>(nb, FR, Ar, fmax);
        TCSCF_LAUNCH(ctx);
        double hm[2];
        TCSCF_CUDA(ctx, cudaMemcpyAsync(hm, fmax, 2 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
        TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (!(hm[0] == hm[0]) || !(hm[1] == hm[1])) return fail(ctx, TCSCF_ERR_NONFINITE, "non-finite Fock matrix");
        if (hm[1] <= 1e-10 * hm[0]) {
          TCSCF_CUDA(ctx, cudaMemcpyAsync(Br, SRre, sizeof(double) * nn, cudaMemcpyDeviceToDevice, ctx->stream));
          if (cusolverDnDsygvd(ctx->solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, nb, Ar, nb, Br, nb, W + s * nb,
                               static_cast<double *>(wkR), lworkR, devInfo) != CUSOLVER_STATUS_SUCCESS)
            return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnDsygvd failed");
          int info = 0;
          TCSCF_CUDA(ctx, cudaMemcpyAsync(&info, devInfo, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
          TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
          if (info != 0) return fail(ctx, TCSCF_ERR_LINALG, "generalized eigen-solve failed (info " + std::to_string(info) + ")");
          kRealDensity<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, nocc[s], Ar, DRre);
          TCSCF_LAUNCH(ctx);
          kRealToReference<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(1, nb, g1->dsto, DRre, nullptr, dD + s * nn);
          TCSCF_LAUNCH(ctx);
          // the next build factors this density as its occupied orbitals themselves (D_R = C C^T):
          // smooth from one iteration to the next, unlike a pivoted factorisation of D
          if (nocc[s] > 0) {
            kFactorFromOrbitals<<<gridBlocks(int64_t(nb) * nocc[s], 256), 256, 0, ctx->stream>>>(nb, nocc[s], Ar, nb, Xocc + size_t(s) * nn);
            TCSCF_LAUNCH(ctx);
            given[s].R = nocc[s];
            given[s].X1 = given[s].X2 = Xocc + size_t(s) * nn;
            given[s].ldx = nb;
            given[s].complex = false;
            given[s].same = true;
          }
          ++solvedReal;
          continue;
        }
      }
      kToColumnMajor<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, Fuse + s * nn, dS, A, B);
      TCSCF_LAUNCH(ctx);
      if (cusolverDnZhegvd(ctx->solver, CUSOLVER_EIG_TYPE_1, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_UPPER, nb,
                           reinterpret_cast<cuDoubleComplex *>(A), nb, reinterpret_cast<cuDoubleComplex *>(B), nb, W + s * nb,
                           static_cast<cuDoubleComplex *>(wk), lwork, devInfo) != CUSOLVER_STATUS_SUCCESS)
        return fail(ctx, TCSCF_ERR_LINALG, "cusolverDnZhegvd failed");
      int info = 0;
      TCSCF_CUDA(ctx, cudaMemcpyAsync(&info, devInfo, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      TCSCF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      if (info != 0) return fail(ctx, TCSCF_ERR_LINALG, "generalized eigen-solve failed (info " + std::to_string(info) + ")");
      kDensityFromOrbitals<<<gridBlocks(nn, 256), 256, 0, ctx->stream>>>(nb, nocc[s], A, dD + s * nn);
      TCSCF_LAUNCH(ctx);
    }
    givenOk = solvedReal == nspin;
  }
  if (energy) *energy = e;
  if (density) TCSCF_CUDA(ctx, cudaMemcpy(density, dD, sizeof(double2) * nn * nspin, cudaMemcpyDeviceToHost));
  if (eigenvalues) TCSCF_CUDA(ctx, cudaMemcpy(eigenvalues, W, sizeof(double) * nb * nspin, cudaMemcpyDeviceToHost));
  return fail(ctx, TCSCF_ERR_NOT_CONVERGED, "Did not converge.");
}

int tcscf_scf_graph(tcscf_ctx * ctx, int r1, int r2, int n_up, int n_down, const double * S, const double * h, int respect_symmetry,
                    int precision, double tol, int max_iter, int capture, double * energy, int * iterations, double * density,
                    double * eigenvalues, int * graph_launches)
{
  TCSCF_NVTX();
  if (!ctx) return TCSCF_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  Grid * g1 = findGrid(ctx, r1);
  Grid * g2 = findGrid(ctx, r2);
  TCSCF_TRY(checkBasisPair(ctx, g1, g2));
  TCSCF_CHECK(ctx, S && h && max_iter > 0, TCSCF_ERR_INVALID_ARGUMENT, "S, h and max_iter are required");
  TCSCF_CHECK(ctx, (n_up + n_down) % 2 == 0 && n_up == n_down, TCSCF_ERR_INVALID_ARGUMENT, "the graph SCF is restricted closed shell");
  TCSCF_CHECK(ctx, precision >= TCSCF_PREC_FP64 && precision <= TCSCF_PREC_TF32, TCSCF_ERR_INVALID_ARGUMENT, "unknown precision");
  int launches = 0;
  int const st = scfGraph(ctx, *g1, *g2, (n_up + n_down) / 2, S, h, respect_symmetry, precision, tol, max_iter, capture, energy, iterations,
                          density, eigenvalues, &launches);
  if (graph_launches) *graph_launches = launches;
  return st;
}

}  // extern "C"
