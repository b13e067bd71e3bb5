// gba_triangulate.cu -- gba_triangulate(): batched multi-view triangulation
// (hs_sfm triangulate/multiple_view_*), FP64.
//
// Each point: undistort its keys (sfm_utility/undistortor.hpp:24-80), build
// the DLT system rows u P3 - P1, v P3 - P2 of P = K [R | -R C]
// (triangulate/multiple_view_dlt.hpp:27-52) as the 4x4 normal matrix
// A^T A, take the eigenvector of its smallest eigenvalue (the smallest right
// singular vector of A), then refine the point by Levenberg-Marquardt (Madsen,
// Nielsen & Tingleff 2004, Alg. 3.16: the driver the reference's
// MultipleViewLevenbergMarquardtOptimizor binds,
// multiple_view_levenberg_marquardt_optimizor.hpp:50-99) on its keys with
// identity weights and the analytical 2x3 point Jacobian of the projection
// (sfm_utility/projective_functions.hpp:22-52).  Tracks are independent, so
// one launch covers the whole batch; the views (36 doubles each, with P and
// the reciprocals of the focal lengths) are expanded once by a small kernel
// and read through the L1.
//
// Bound by the FP64 pipe (64 cycles an instruction and warp, whatever its
// lanes do), which decides the layout:
//  - a large batch runs one thread per track, the tracks ordered by their
//    length (tri_order), so that a warp's lanes have the same number of views
//    (2 to 12 views: the longest of 32 is 12, the mean 7);
//  - a batch that does not fill the schedulers' lanes twice runs 2, 4 or 8
//    lanes per track, which share its views and its sums' entries (RowSums):
//    its time is one warp's instruction count;
//  - the candidate's cost and normal equations are formed in one pass (nearly
//    every step is accepted), and the eigenvector comes from inverse iteration
//    (about 200 instructions) instead of Jacobi sweeps (about 3,300), which
//    remain for the systems where it does not settle.
// 1M tracks of 2 to 12 views 24.3 -> 7.3 ms, 40,000 tracks 1.44 -> 0.47 ms,
// 3,001 tracks of 2 to 8 views 0.41 -> 0.095 ms.
#include "gba_internal.h"

#include <cmath>
#include <cstdio>
#include <vector>

namespace gba {
namespace {

#define TRI_CUDA(call)                                                          \
  do {                                                                          \
    cudaError_t e_ = (call);                                                    \
    if (e_ != cudaSuccess) {                                                    \
      std::fprintf(stderr, "gba: %s failed: %s\n", #call, cudaGetErrorString(e_)); \
      throw CudaError{e_ == cudaErrorMemoryAllocation ? GBA_ERR_OOM : GBA_ERR_CUDA}; \
    }                                                                           \
  } while (0)

// f s cx cy f*a k1 k2 k3 d1 d2, R (9), C (3), P = K [R | -R C] (12), 1/f, 1/(f a)
constexpr int kViewDoubles = 36;

thread_local double g_tri_last_ms = 0.0;   // the calling thread's last kernel time (profile)

__global__ void k_tri_views(int V, const double* __restrict__ intr, const double* __restrict__ extr,
                            double* __restrict__ views) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  double* o = views + (long long)kViewDoubles * v;
  for (int j = 0; j < 10; ++j) o[j] = intr[10LL * v + j];
  const double f = o[0], s = o[1], cx = o[2], cy = o[3], fa = o[0] * o[4];
  o[4] = fa;
  const double r0 = extr[6LL * v], r1 = extr[6LL * v + 1], r2 = extr[6LL * v + 2];
  const double th = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
  double* R = o + 10;
  if (th == 0.0) {
    for (int j = 0; j < 9; ++j) R[j] = (j % 4 == 0) ? 1.0 : 0.0;
  } else {   // world to camera: cos I + sin [k]x + (1 - cos) k k^T
    const double k0 = r0 / th, k1 = r1 / th, k2 = r2 / th;
    const double c = cos(th), sn = sin(th), t = 1.0 - c;
    R[0] = c + t * k0 * k0;       R[1] = t * k0 * k1 - sn * k2; R[2] = t * k0 * k2 + sn * k1;
    R[3] = t * k1 * k0 + sn * k2; R[4] = c + t * k1 * k1;       R[5] = t * k1 * k2 - sn * k0;
    R[6] = t * k2 * k0 - sn * k1; R[7] = t * k2 * k1 + sn * k0; R[8] = c + t * k2 * k2;
  }
  double* C = o + 19;
  for (int j = 0; j < 3; ++j) C[j] = extr[6LL * v + 3 + j];
  double Rt[12];   // [R | -R C]
  for (int r = 0; r < 3; ++r) {
    for (int c = 0; c < 3; ++c) Rt[4 * r + c] = R[3 * r + c];
    Rt[4 * r + 3] = -(R[3 * r] * C[0] + R[3 * r + 1] * C[1] + R[3 * r + 2] * C[2]);
  }
  double* P = o + 22;
  for (int c = 0; c < 4; ++c) {
    P[c] = f * Rt[c] + s * Rt[4 + c] + cx * Rt[8 + c];
    P[4 + c] = fa * Rt[4 + c] + cy * Rt[8 + c];
    P[8 + c] = Rt[8 + c];
  }
  o[34] = 1.0 / f;
  o[35] = 1.0 / fa;
}

// N doubles from a 16-byte aligned address.
template <int N>
__device__ __forceinline__ void ld2(const double* __restrict__ p, double* o) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p + i));
    o[i] = v.x;
    o[i + 1] = v.y;
  }
}

// The sums over a track's views of two rows' products, in the views' order
// whatever G, so a track has the same bits in any batch.  Each view gives two
// rows of four values; entry e of the sums is the e-th (r, c), r <= c, of the
// 4 x 4 upper triangle: sum += ra[r] ra[c], then rb[r] rb[c].  A group's lanes
// form the rows of G views at a time; its entries are shared out over the
// lanes, which read the rows one after the other from shared memory: of the
// FP64 pipe's instructions only 2 to 10 a view instead of 20.  (Sums added by
// shuffles in a tree cost the same, 0.097 ms against 0.095 for 3,001 tracks,
// but a track's last digits then changed with the size of its batch.)
template <int G>
struct RowSums {
  static constexpr int kOwn = (10 + G - 1) / G;
  double acc[kOwn];
  double (*buf)[8];   // the group's rows [G][8] (G > 1)
  int sub;
  unsigned mask;

  __device__ __forceinline__ RowSums(double (*rows)[8], int sub_, unsigned mask_)
      : buf(G > 1 ? rows + threadIdx.x / G * G : rows), sub(sub_), mask(mask_) {
#pragma unroll
    for (int u = 0; u < kOwn; ++u) acc[u] = 0.0;
  }
  static __device__ __forceinline__ int row(int e) { return e < 4 ? 0 : e < 7 ? 1 : e < 9 ? 2 : 3; }
  static __device__ __forceinline__ int col(int e) { return e < 4 ? e : e < 7 ? e - 3 : e < 9 ? e - 5 : 3; }
  // The rows of the next `views` (at most G) views, the sub-th of them this lane's.
  __device__ __forceinline__ void add(const double ra[4], const double rb[4], int views) {
    if constexpr (G == 1) {
#pragma unroll
      for (int e = 0; e < 10; ++e) acc[e] = fma(rb[row(e)], rb[col(e)], fma(ra[row(e)], ra[col(e)], acc[e]));
    } else {
      __syncwarp(mask);   // (the last rows are read)
      if (sub < views) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          buf[sub][c] = ra[c];
          buf[sub][4 + c] = rb[c];
        }
      }
      __syncwarp(mask);
      for (int l = 0; l < views; ++l) {
#pragma unroll
        for (int u = 0; u < kOwn; ++u) {
          const int e = min(sub + G * u, 9);
          const double* v = buf[l];
          acc[u] = fma(v[4 + row(e)], v[4 + col(e)], fma(v[row(e)], v[col(e)], acc[u]));
        }
      }
    }
  }
  // Every lane gets the ten sums.
  __device__ __forceinline__ void get(double s[10]) {
    if constexpr (G == 1) {
#pragma unroll
      for (int e = 0; e < 10; ++e) s[e] = acc[e];
    } else {
      double* all = buf[0];
      __syncwarp(mask);
#pragma unroll
      for (int u = 0; u < kOwn; ++u)
        if (sub + G * u < 10) all[sub + G * u] = acc[u];
      __syncwarp(mask);
#pragma unroll
      for (int e = 0; e < 10; ++e) s[e] = all[e];
    }
  }
};

// Normal matrix, gradient and cost of a track at X: s = (N00 N01 N02 g0 N11
// N12 g1 N22 g2 F), the upper triangle of the sums over (J, residual).
template <int G>
__device__ __forceinline__ void tri_normal(const double* __restrict__ views, const long long* __restrict__ tv,
                                           const double* __restrict__ keys, int m, int sub, unsigned mask,
                                           double (*rows)[8], const double X[3], double s[10]) {
  RowSums<G> sums(rows, sub, mask);
  for (int base = 0; base < m; base += G) {
    const int i = base + sub;
    double J[2][4] = {};   // (d key / d X, residual) of u and v
    if (i < m) {
      double w[22];   // f s cx cy fa k1 k2 k3 d1 d2 R C
      ld2<22>(views + kViewDoubles * tv[i], w);
      const double* R = w + 10;
      const double e0 = X[0] - w[19], e1 = X[1] - w[20], e2 = X[2] - w[21];
      const double c0 = fma(R[2], e2, fma(R[1], e1, R[0] * e0));
      const double c1 = fma(R[5], e2, fma(R[4], e1, R[3] * e0));
      const double c2 = fma(R[8], e2, fma(R[7], e1, R[6] * e0));
      const double iz = 1.0 / c2;
      const double x = c0 * iz, y = c1 * iz;
      const double r2 = fma(y, y, x * x);
      const double k1 = w[5], k2 = w[6], k3 = w[7], d1 = w[8], d2 = w[9];
      const double c = r2 * fma(r2, fma(r2, k3, k2), k1);
      const double x2 = x + x, y2 = y + y, xy2 = x2 * y;
      const double ex = fma(d1, xy2, fma(d2, fma(x2, x, r2), fma(c, x, x)));
      const double ey = fma(d2, xy2, fma(d1, fma(y2, y, r2), fma(c, y, y)));
      const double f = w[0], sk = w[1], fa = w[4];
      J[0][3] = fma(f, ex, fma(sk, ey, w[2])) - keys[2 * i];
      J[1][3] = fma(fa, ey, w[3]) - keys[2 * i + 1];
      // d key / d (x, y), then by the camera point (b), then by X
      const double dc = 2.0 * fma(r2, fma(r2, 3.0 * k3, 2.0 * k2), k1);
      const double t = dc * x, q = 1.0 + c;
      const double exx = fma(t, x, fma(d1, y2, fma(3.0 * d2, x2, q)));
      const double exy = fma(t, y, fma(d1, x2, d2 * y2));
      const double eyy = fma(dc * y, y, fma(d2, x2, fma(3.0 * d1, y2, q)));
      const double bx[2] = {fma(f, exx, sk * exy) * iz, fa * exy * iz};
      const double by[2] = {fma(f, exy, sk * eyy) * iz, fa * eyy * iz};
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const double bz = -fma(bx[r], x, by[r] * y);
#pragma unroll
        for (int j = 0; j < 3; ++j) J[r][j] = fma(bz, R[6 + j], fma(by[r], R[3 + j], bx[r] * R[j]));
      }
    }
    sums.add(J[0], J[1], min(G, m - base));
  }
  sums.get(s);
}

// (N + mu I) d = g (of tri_normal's sums) by a 3x3 Cholesky; false when not
// positive definite.
__device__ __forceinline__ bool tri_solve(const double s[10], double mu, double d[3]) {
  const double N[6] = {s[0], s[1], s[2], s[4], s[5], s[7]}, g[3] = {s[3], s[6], s[8]};
  const double a00 = N[0] + mu, a11 = N[3] + mu, a22 = N[5] + mu;
  if (!(a00 > 0.0)) return false;
  const double i0 = rsqrt(a00), l10 = N[1] * i0, l20 = N[2] * i0;
  const double s11 = fma(-l10, l10, a11);
  if (!(s11 > 0.0)) return false;
  const double i1 = rsqrt(s11), l21 = fma(-l20, l10, N[4]) * i1;
  const double s22 = fma(-l21, l21, fma(-l20, l20, a22));
  if (!(s22 > 0.0)) return false;
  const double i2 = rsqrt(s22);
  const double y0 = g[0] * i0, y1 = fma(-l10, y0, g[1]) * i1, y2 = fma(-l21, y1, fma(-l20, y0, g[2])) * i2;
  d[2] = y2 * i2;
  d[1] = fma(-l21, d[2], y1) * i1;
  d[0] = fma(-l20, d[2], fma(-l10, d[1], y0)) * i0;
  return true;
}

// Eigenvector of the smallest eigenvalue of the symmetric 4x4 A (row-major),
// cyclic Jacobi (Golub & Van Loan 8.5), at most 30 sweeps.
__device__ __noinline__ void tri_jacobi(double A[16], double out[4]) {
  double V[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) V[e] = (e % 5 == 0) ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 30; ++sweep) {
    double off = 0.0, tot = 0.0;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      tot += A[e] * A[e];
      if (e % 5 != 0) off += A[e] * A[e];
    }
    if (off <= 1e-30 * tot) break;
#pragma unroll
    for (int p = 0; p < 3; ++p) {
#pragma unroll
      for (int q = p + 1; q < 4; ++q) {
        const double apq = A[4 * p + q];
        if (apq != 0.0) {
          const double theta = (A[4 * q + q] - A[4 * p + p]) / (2.0 * apq);
          const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
          const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double akp = A[4 * k + p], akq = A[4 * k + q];
            A[4 * k + p] = c * akp - s * akq;
            A[4 * k + q] = s * akp + c * akq;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double apk = A[4 * p + k], aqk = A[4 * q + k];
            A[4 * p + k] = c * apk - s * aqk;
            A[4 * q + k] = s * apk + c * aqk;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const double vkp = V[4 * k + p], vkq = V[4 * k + q];
            V[4 * k + p] = c * vkp - s * vkq;
            V[4 * k + q] = s * vkp + c * vkq;
          }
        }
      }
    }
  }
  double best = A[0];
#pragma unroll
  for (int k = 0; k < 4; ++k) out[k] = V[4 * k];
#pragma unroll
  for (int i = 1; i < 4; ++i)
    if (A[5 * i] < best) {
      best = A[5 * i];
#pragma unroll
      for (int k = 0; k < 4; ++k) out[k] = V[4 * k + i];
    }
}

// The same by inverse iteration on A = L D L^T (Golub & Van Loan 8.2.2): A is
// a sum of squares, so the unpivoted factorization is stable, and the
// error falls by (smallest / next eigenvalue) a step.  M: the upper triangle,
// rows.  Rank below three (no unique vector), no positive pivots, no settling
// in 16 steps (the two smallest eigenvalues close), or an eigenvalue below the
// one found: Jacobi.  The last is a vector without a homogeneous coordinate (a
// point at infinity), of which the start has no part.  It is ruled out when
// the leading 3 x 3 block has no eigenvalue at or below the one found: the
// second smallest of A is not below that block's smallest.
__device__ __forceinline__ void tri_smallest_eigenvector(const double M[10], double x[4]) {
  const double trace = M[0] + M[4] + M[7] + M[9];
  const double tiny = 1e-13 * trace;
  const double d0 = M[0], i0 = 1.0 / d0;
  const double l10 = M[1] * i0, l20 = M[2] * i0, l30 = M[3] * i0;
  const double d1 = fma(-l10, M[1], M[4]), a21 = fma(-l10, M[2], M[5]), a31 = fma(-l10, M[3], M[6]);
  const double i1 = 1.0 / d1, l21 = a21 * i1, l31 = a31 * i1;
  const double d2 = fma(-l21, a21, fma(-l20, M[2], M[7]));
  const double a32 = fma(-l21, a31, fma(-l20, M[3], M[8]));
  const double i2 = 1.0 / d2, l32 = a32 * i2;
  const double e3 = fma(-l32, a32, fma(-l31, a31, fma(-l30, M[3], M[9])));
  bool settled = false;
  if (d0 > tiny && d1 > tiny && d2 > tiny) {
    // (exact data leaves rounding for a last pivot)
    const double i3 = 1.0 / fmax(e3, 1e-18 * trace);
    // start: L^T x = e3, the limit of a vanishing last pivot
    x[3] = 1.0;
    x[2] = -l32;
    x[1] = -fma(l21, x[2], l31);
    x[0] = -fma(l10, x[1], fma(l20, x[2], l30));
    double r = rsqrt(fma(x[3], x[3], fma(x[2], x[2], fma(x[1], x[1], x[0] * x[0]))));
#pragma unroll
    for (int e = 0; e < 4; ++e) x[e] *= r;
    for (int it = 0; it < 16 && !settled; ++it) {
      double y[4];
      y[0] = x[0];
      y[1] = fma(-l10, y[0], x[1]);
      y[2] = fma(-l21, y[1], fma(-l20, y[0], x[2]));
      y[3] = fma(-l32, y[2], fma(-l31, y[1], fma(-l30, y[0], x[3]))) * i3;
      y[2] = fma(-l32, y[3], y[2] * i2);
      y[1] = fma(-l31, y[3], fma(-l21, y[2], y[1] * i1));
      y[0] = fma(-l30, y[3], fma(-l20, y[2], fma(-l10, y[1], y[0] * i0)));
      r = rsqrt(fma(y[3], y[3], fma(y[2], y[2], fma(y[1], y[1], y[0] * y[0]))));
      double diff = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double z = y[e] * r, dz = z - x[e];
        diff = fma(dz, dz, diff);
        x[e] = z;
      }
      settled = diff <= 1e-29;
    }
    // the block less the eigenvalue r is positive definite: its leading minors
    // (m3: the determinant times a00)
    const double l = r * (1.0 + 1e-9), a00 = M[0] - l, a11 = M[4] - l, a22 = M[7] - l;
    const double m2 = fma(-M[1], M[1], a00 * a11), c12 = fma(a00, M[5], -(M[1] * M[2]));
    const double m3 = fma(-c12, c12, m2 * fma(-M[2], M[2], a00 * a22));
    settled = settled && a00 > 0.0 && m2 > 0.0 && m3 > 0.0;
  }
  if (!settled) {
    double A[16] = {M[0], M[1], M[2], M[3], M[1], M[4], M[5], M[6],
                    M[2], M[5], M[7], M[8], M[3], M[6], M[8], M[9]};
    tri_jacobi(A, x);
  }
}

struct TriParams {
  int max_iterations;
  double tau, eps1, eps2;
};

// G lanes per track; order (or null): the track of each group.
template <int G>
__global__ void __launch_bounds__(128) k_triangulate(long long n, const int* __restrict__ order,
                                                     const long long* __restrict__ off,
                                                     const long long* __restrict__ track_views,
                                                     const double* __restrict__ track_keys,
                                                     const double* __restrict__ views, TriParams prm,
                                                     double* __restrict__ points, int* __restrict__ status) {
  __shared__ double rows[G > 1 ? 128 : 1][8];
  const long long slot = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / G;
  if (slot >= n) return;
  const int sub = threadIdx.x % G;
  const unsigned mask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << ((threadIdx.x & 31) / G * G);
  const long long j = order ? order[slot] : slot;
  const long long t0 = off[j];
  const int m = int(off[j + 1] - t0);
  const long long* tv = track_views + t0;
  const double* keys = track_keys + 2 * t0;
  double X[3] = {0.0, 0.0, 0.0};
  int st = GBA_OK;
  if (m < 2) {
    st = GBA_ERR_INVALID;
  } else {
    // DLT normal matrix A^T A (upper triangle) of the undistorted keys
    RowSums<G> sums(rows, sub, mask);
    for (int base = 0; base < m; base += G) {
      const int i = base + sub;
      double a[4] = {}, b[4] = {};
      if (i < m) {
        const double* vw = views + kViewDoubles * tv[i];
        double w[10], P[14];
        ld2<10>(vw, w);
        ld2<14>(vw + 22, P);   // P, 1 / f, 1 / (f a)
        const double k1 = w[5], k2 = w[6], k3 = w[7], d1 = w[8], d2 = w[9];
        const double y0 = (keys[2 * i + 1] - w[3]) * P[13];
        const double x0 = fma(-w[1], y0, keys[2 * i] - w[2]) * P[12];
        double x = x0, y = y0;
        for (int it = 0; it < 5; ++it) {
          const double r2 = fma(y, y, x * x);
          const double rc = 1.0 / fma(r2, fma(r2, fma(r2, k3, k2), k1), 1.0);
          const double x2 = x + x, xy2 = x2 * y;
          const double dx = fma(d1, xy2, d2 * fma(x2, x, r2));
          const double dy = fma(d2, xy2, d1 * fma(y + y, y, r2));
          x = (x0 - dx) * rc;
          y = (y0 - dy) * rc;
        }
        const double u = fma(w[0], x, fma(w[1], y, w[2])), v = fma(w[4], y, w[3]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          a[c] = fma(u, P[8 + c], -P[c]);
          b[c] = fma(v, P[8 + c], -P[4 + c]);
        }
      }
      sums.add(a, b, min(G, m - base));
    }
    double M[10];
    sums.get(M);
    double h[4];
    tri_smallest_eigenvector(M, h);
    if (h[3] == 0.0) {
      st = GBA_ERR_NAN;
    } else {
      X[0] = h[0] / h[3];
      X[1] = h[1] / h[3];
      X[2] = h[2] / h[3];
      if (!(isfinite(X[0]) && isfinite(X[1]) && isfinite(X[2]))) st = GBA_ERR_NAN;
    }
    if (st == GBA_OK) {   // LM refinement
      double s[10];
      tri_normal<G>(views, tv, keys, m, sub, mask, rows, X, s);
      auto gradient = [&] { return fmax(fabs(s[3]), fmax(fabs(s[6]), fabs(s[8]))); };
      bool found = gradient() <= prm.eps1;
      double mu = prm.tau * fmax(s[0], fmax(s[4], s[7]));
      double nu = 2.0;
      for (int k = 0; !found && k < prm.max_iterations; ++k) {
        double d[3];
        if (!tri_solve(s, mu, d)) {
          mu *= nu;
          nu *= 2.0;
          continue;
        }
        const double dn2 = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
        const double xn = sqrt(fma(X[2], X[2], fma(X[1], X[1], X[0] * X[0])));
        if (sqrt(dn2) <= prm.eps2 * (xn + prm.eps2)) break;
        const double Xn[3] = {X[0] - d[0], X[1] - d[1], X[2] - d[2]};
        double sn[10];
        tri_normal<G>(views, tv, keys, m, sub, mask, rows, Xn, sn);
        const double denom = fma(mu, dn2, fma(s[8], d[2], fma(s[6], d[1], s[3] * d[0])));
        const double rho = (s[9] - sn[9]) / denom;
        if (isfinite(sn[9]) && rho > 0.0) {
#pragma unroll
          for (int e = 0; e < 3; ++e) X[e] = Xn[e];
#pragma unroll
          for (int e = 0; e < 10; ++e) s[e] = sn[e];
          found = gradient() <= prm.eps1;
          const double tt = 2.0 * rho - 1.0;
          mu *= fmax(1.0 / 3.0, 1.0 - tt * tt * tt);
          nu = 2.0;
        } else {
          mu *= nu;
          nu *= 2.0;
        }
      }
      if (!isfinite(s[9])) st = GBA_ERR_NAN;
    }
  }
  if (sub < 3) points[3 * j + sub] = sub == 0 ? X[0] : sub == 1 ? X[1] : X[2];
  if (G < 3 && sub == 0) {   // (fewer lanes than coordinates)
    if (G < 2) points[3 * j + 1] = X[1];
    points[3 * j + 2] = X[2];
  }
  if (sub == 0) status[j] = st;
}

// The tracks by descending length (any order within one length: a track's
// result does not depend on its place).  bins [2 * kTriBins]: counts, then
// each length's next place.
constexpr int kTriBins = 64;

__device__ __forceinline__ int tri_bin(const long long* off, long long j) {
  const long long m = off[j + 1] - off[j];
  return kTriBins - 1 - int(m < kTriBins ? m : kTriBins - 1);   // longest first
}

__global__ void __launch_bounds__(256) k_tri_count(long long n, const long long* __restrict__ off, int* bins) {
  __shared__ int h[kTriBins];
  if (threadIdx.x < kTriBins) h[threadIdx.x] = 0;
  __syncthreads();
  const long long j = blockIdx.x * 256LL + threadIdx.x;
  if (j < n) atomicAdd(&h[tri_bin(off, j)], 1);
  __syncthreads();
  if (threadIdx.x < kTriBins && h[threadIdx.x] > 0) atomicAdd(bins + threadIdx.x, h[threadIdx.x]);
}

__global__ void __launch_bounds__(kTriBins) k_tri_places(int* bins) {
  int run = 0;
  for (int b = 0; b < int(threadIdx.x); ++b) run += bins[b];
  bins[kTriBins + threadIdx.x] = run;
}

__global__ void __launch_bounds__(256) k_tri_order(long long n, const long long* __restrict__ off, int* bins,
                                                   int* __restrict__ order) {
  __shared__ int h[kTriBins], base[kTriBins];
  if (threadIdx.x < kTriBins) h[threadIdx.x] = 0;
  __syncthreads();
  const long long j = blockIdx.x * 256LL + threadIdx.x;
  const int b = j < n ? tri_bin(off, j) : 0;
  const int rank = j < n ? atomicAdd(&h[b], 1) : 0;
  __syncthreads();
  if (threadIdx.x < kTriBins && h[threadIdx.x] > 0)
    base[threadIdx.x] = atomicAdd(bins + kTriBins + threadIdx.x, h[threadIdx.x]);
  __syncthreads();
  if (j < n) order[base[b] + rank] = int(j);
}

}  // namespace
}  // namespace gba

extern "C" int gba_triangulate(const gba_triangulation* p, const gba_options* o, double* points,
                               int32_t* point_status) {
  using namespace gba;
  if (!p || !o || !points || p->number_of_views < 0 || p->number_of_points < 0 ||
      o->max_iterations < 0)
    return GBA_ERR_INVALID;
  const long long V = p->number_of_views, n = p->number_of_points;
  if (n == 0) return GBA_OK;
  if (!p->track_offsets || (V > 0 && (!p->intrinsics || !p->extrinsics))) return GBA_ERR_INVALID;
  if (p->track_offsets[0] != 0) return GBA_ERR_INVALID;
  for (long long j = 0; j < n; ++j)
    if (p->track_offsets[j + 1] < p->track_offsets[j]) return GBA_ERR_INVALID;
  const long long m = p->track_offsets[n];
  if (m > 0 && (!p->track_views || !p->track_keys)) return GBA_ERR_INVALID;
  for (long long t = 0; t < m; ++t)
    if (p->track_views[t] < 0 || p->track_views[t] >= V) return GBA_ERR_BAD_INDEX;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return GBA_ERR_NO_DEVICE;
  }
  cudaStream_t s = nullptr;
  std::vector<void*> bufs;
  int err = GBA_OK;
  try {
    TRI_CUDA(cudaSetDevice(o->device));
    TRI_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    auto dev = [&](size_t bytes) {
      void* d = nullptr;
      TRI_CUDA(cudaMallocAsync(&d, bytes > 0 ? bytes : 1, s));
      bufs.push_back(d);
      return d;
    };
    auto up = [&](const void* h, size_t bytes) {
      void* d = dev(bytes);
      if (bytes) TRI_CUDA(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s));
      return d;
    };
    const double* d_intr = static_cast<const double*>(up(p->intrinsics, sizeof(double) * 10 * V));
    const double* d_extr = static_cast<const double*>(up(p->extrinsics, sizeof(double) * 6 * V));
    double* d_views = static_cast<double*>(dev(sizeof(double) * kViewDoubles * (V > 0 ? V : 1)));
    const long long* d_off = static_cast<const long long*>(up(p->track_offsets, sizeof(int64_t) * (n + 1)));
    const long long* d_tv = static_cast<const long long*>(up(p->track_views, sizeof(int64_t) * m));
    const double* d_keys = static_cast<const double*>(up(p->track_keys, sizeof(double) * 2 * m));
    double* d_pts = static_cast<double*>(dev(sizeof(double) * 3 * n));
    int* d_st = static_cast<int*>(dev(sizeof(int) * n));
    int launches = 0;
    if (V > 0) {
      k_tri_views<<<unsigned((V + 127) / 128), 128, 0, s>>>(int(V), d_intr, d_extr, d_views);
      ++launches;
    }
    TriParams prm{o->max_iterations, o->tau, o->eps1, o->eps2};
    cudaEvent_t ev[2] = {nullptr, nullptr};
    if (o->profile) {
      TRI_CUDA(cudaEventCreate(&ev[0]));
      TRI_CUDA(cudaEventCreate(&ev[1]));
      TRI_CUDA(cudaEventRecord(ev[0], s));
    }
    // lanes per track: while the batch leaves lanes of the schedulers (four
    // warps an SM) idle twice over; one thread per track above, ordered by
    // length (n <= INT32_MAX: the order's indices)
    int sms = 0;
    TRI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, o->device));
    const long long lanes = 2LL * 4 * sms * 32;
    const int G = n * 8 <= lanes ? 8 : n * 4 <= lanes ? 4 : n * 2 <= lanes ? 2 : 1;
    int* d_order = nullptr;
    if (G == 1 && n <= INT32_MAX) {
      int* bins = static_cast<int*>(dev(sizeof(int) * 2 * kTriBins));
      d_order = static_cast<int*>(dev(sizeof(int) * n));
      const unsigned gn = unsigned((n + 255) / 256);
      TRI_CUDA(cudaMemsetAsync(bins, 0, sizeof(int) * kTriBins, s));
      k_tri_count<<<gn, 256, 0, s>>>(n, d_off, bins);
      k_tri_places<<<1, kTriBins, 0, s>>>(bins);
      k_tri_order<<<gn, 256, 0, s>>>(n, d_off, bins, d_order);
      launches += 3;
    }
    const unsigned g = unsigned((n * G + 127) / 128);
    switch (G) {
      case 8: k_triangulate<8><<<g, 128, 0, s>>>(n, d_order, d_off, d_tv, d_keys, d_views, prm, d_pts, d_st); break;
      case 4: k_triangulate<4><<<g, 128, 0, s>>>(n, d_order, d_off, d_tv, d_keys, d_views, prm, d_pts, d_st); break;
      case 2: k_triangulate<2><<<g, 128, 0, s>>>(n, d_order, d_off, d_tv, d_keys, d_views, prm, d_pts, d_st); break;
      default: k_triangulate<1><<<g, 128, 0, s>>>(n, d_order, d_off, d_tv, d_keys, d_views, prm, d_pts, d_st);
    }
    ++launches;
    TRI_CUDA(cudaGetLastError());
    g_tri_last_ms = 0.0;
    if (o->profile) {
      TRI_CUDA(cudaEventRecord(ev[1], s));
      TRI_CUDA(cudaEventSynchronize(ev[1]));
      float ms = 0.0f;
      TRI_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      g_tri_last_ms = ms;
      cudaEventDestroy(ev[0]);
      cudaEventDestroy(ev[1]);
    }
    count_launches(launches);
    TRI_CUDA(cudaMemcpyAsync(points, d_pts, sizeof(double) * 3 * n, cudaMemcpyDeviceToHost, s));
    std::vector<int> st(static_cast<size_t>(n));
    TRI_CUDA(cudaMemcpyAsync(st.data(), d_st, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
    TRI_CUDA(cudaStreamSynchronize(s));
    if (point_status)
      for (long long j = 0; j < n; ++j) point_status[j] = st[size_t(j)];
  } catch (const CudaError& e) {
    err = e.status;
  }
  for (void* b : bufs) cudaFreeAsync(b, s);
  if (s) {
    cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
  }
  return err;
}

extern "C" double gba_triangulate_last_kernel_ms(void) { return gba::g_tri_last_ms; }
