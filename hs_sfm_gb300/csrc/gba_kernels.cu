// gba_kernels.cu -- the sm_103a kernels of one Levenberg-Marquardt iteration
// over a batch of bundle-adjustment problems, and their launchers.
//
// Stage map (reference: include/hs_sfm/bundle_adjustment/):
//   k_image_prep     rotation of each image: Rodrigues matrix (FP64) and the
//                    coefficients of the analytical rotation derivative
//                    (camera_shared_analytical_jacobian_matrix_calculator.hpp:341-380)
//   k_cost           r = f(x) - y in FP64, whitening by the key weight, Huber
//                    rho and IRLS weight, per-chunk FP64 cost sums
//                    (camera_shared_vector_function.hpp:634-744,
//                     camera_shared_mahalanobis_distance_calculator.hpp:28-58)
//   k_linearize      per point: analytical Jacobian of each key (T), whitened
//                    blocks J_p, J_i, V_p = sum J_p^T J_p, g_p = sum J_p^T r
//                    (analytical_jacobian_matrix_calculator.hpp:66-557,
//                     normal_equation_builder.hpp:207-220,377-391)
//   k_image_reduce   per image: U_i = sum J_i^T J_i, g_i = sum J_i^T r with
//                    compensated (Kahan) lane sums (normal_equation_builder.hpp:221-234)
//   k_point_factor   per point: C C^T = V_p + mu I, h_p = C^-1 g_p, and
//   k_key_z          per key: Z_a = C^-1 J_p^T J_i (normal_equation_solver.hpp:141-184)
//   k_assemble_items per block (i<=j) of the reduced system: -sum Z_a^T Z_b
//                    over the points seen by both images, rhs terms
//                    (normal_equation_solver.hpp:190-267,398-420)
//   k_assemble_S     dense reduced system S and rhs b (T), block sums in FP64
//   k_chol_*         tiled Cholesky (T) with the forward solve folded in,
//                    then the backward solve (normal_equation_solver.hpp:448-466)
//   k_backsub        delta_p = C^-T (h_p - C^-1 sum J_p^T J_i delta_i), x_new = x - delta,
//                    and the candidate's image rotations
//                    (normal_equation_solver.hpp:468-538)
//   k_ctrl_*         the LM decisions per problem on the device (Madsen,
//                    Nielsen & Tingleff 2004, Alg. 3.16 as bound by
//                    camera_shared_nllso_meta_levenberg_marquardt.hpp:33-106)
//   free cameras:    k_cam_prep (camera arrays of x), J_c in k_linearize_keys,
//                    k_image_cam_reduce / k_image_cam_finalize / k_cam_finalize
//                    (E_i = J_i^T J_c, U_c, g_c), k_camrec_z (camera Z
//                    records), camera parts in k_assemble_S, k_cam_backsub
//                    (normal_equation_builder.hpp:157-205,309-349;
//                     normal_equation_solver.hpp:270-392,422-443)
//   PCG:             k_assemble_blocks, k_pcg_* (block-Jacobi PCG on the
//                    explicit 6x6 blocks of S)
#include "gba_factor_layout.h"
#include "gba_internal.h"

#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstdio>

namespace gba {
namespace {

namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long dbits(double v) {
  return static_cast<unsigned long long>(__double_as_longlong(v));
}
__device__ __forceinline__ double bitsd(unsigned long long b) {
  return __longlong_as_double(static_cast<long long>(b));
}

template <typename T>
__device__ __forceinline__ T ldg(const T* p) { return __ldg(p); }

// Load N consecutive T (N even for double, multiple of 4 for float) from a
// 16-byte aligned address with vector loads.
template <int N>
__device__ __forceinline__ void load_vec(const float* __restrict__ p, float* out) {
  static_assert(N % 4 == 0 || N == 2, "float vectors of 4 (or one float2)");
  if constexpr (N == 2) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    out[0] = v.x;
    out[1] = v.y;
  } else {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) {
      float4 v = __ldg(reinterpret_cast<const float4*>(p) + i);
      out[4 * i] = v.x; out[4 * i + 1] = v.y; out[4 * i + 2] = v.z; out[4 * i + 3] = v.w;
    }
  }
}
template <int N>
__device__ __forceinline__ void load_vec(const double* __restrict__ p, double* out) {
  static_assert(N % 2 == 0, "double vectors of 2");
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    double2 v = __ldg(reinterpret_cast<const double2*>(p) + i);
    out[2 * i] = v.x; out[2 * i + 1] = v.y;
  }
}
template <int N>
__device__ __forceinline__ void store_vec(float* p, const float* in) {
#pragma unroll
  for (int i = 0; i < N / 4; ++i)
    reinterpret_cast<float4*>(p)[i] = make_float4(in[4 * i], in[4 * i + 1], in[4 * i + 2], in[4 * i + 3]);
}
template <int N>
__device__ __forceinline__ void store_vec(double* p, const double* in) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i)
    reinterpret_cast<double2*>(p)[i] = make_double2(in[2 * i], in[2 * i + 1]);
}

// Z records (18 T each) at slot s: either records of kZStride T in slot
// order, or (DevPlan::z_planes) nine planes of T pairs, plane v holding the
// pair (z[2v], z[2v+1]) of every slot (plane stride z_n slots).
template <typename T> struct Pair2;
template <> struct Pair2<float> { using type = float2; };
template <> struct Pair2<double> { using type = double2; };

template <typename T>
__device__ __forceinline__ void load_z(const DevPlan& d, const T* __restrict__ Z, long long s, T* z) {
  if (d.z_planes) {
    const auto* zp = reinterpret_cast<const typename Pair2<T>::type*>(Z) + s;
#pragma unroll
    for (int v = 0; v < 9; ++v) {
      const auto t = __ldg(zp + v * d.z_n);
      z[2 * v] = t.x;
      z[2 * v + 1] = t.y;
    }
  } else {
    load_vec<kZStride>(Z + (long long)kZStride * s, z);
  }
}

template <typename T>
__device__ __forceinline__ void store_z(const DevPlan& d, T* Z, long long s, const T* z) {
  if (d.z_planes) {
    auto* zp = reinterpret_cast<typename Pair2<T>::type*>(Z) + s;
#pragma unroll
    for (int v = 0; v < 9; ++v) zp[v * d.z_n] = {z[2 * v], z[2 * v + 1]};
  } else {
    store_vec<kZStride>(Z + (long long)kZStride * s, z);
  }
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename T>
__device__ __forceinline__ T warp_sum_t(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of N values per lane over the warp, the sums scattered over the lanes:
// each halving step o = 16 .. 1 gives the partner lane half of the values
// still held and adds its half of the others, so a value's sum is formed by
// the same tree as warp_sum_t's (the same bits) with about N additions and
// shuffles in all instead of 5 N.  Lane l ends with the sums of the values
// base .. base + count - 1 in v[0 .. count - 1] (count at most
// warp_scatter_max(N), possibly 0).
__host__ __device__ constexpr int warp_scatter_max(int n) {
  for (int o = 16; o > 0; o >>= 1) n = (n + 1) / 2;
  return n;
}
// kLast: the levels below it are left to the caller.
template <int N, int O = 16, int kLast = 1, typename T>
__device__ __forceinline__ void warp_scatter_sums(T* v, int lane, int& base, int& count) {
  if constexpr (O == 16) {
    base = 0;
    count = N;
  }
  if constexpr (O >= kLast) {
    constexpr int H = (N + 1) / 2;
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int i = 0; i < H; ++i) {
      const T hi = H + i < N ? v[H + i < N ? H + i : i] : T(0);
      const T keep = up ? hi : v[i], give = up ? v[i] : hi;
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
    }
    base += up ? H : 0;
    count = up ? count - H : min(count, H);
    warp_scatter_sums<H, O / 2, kLast, T>(v, lane, base, count);
  }
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Deterministic block sum of one double per thread (blockDim multiple of 32,
// at most 1024).  Result valid in thread 0.
__device__ double block_sum(double v, double* smem) {
  v = warp_sum(v);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) smem[w] = v;
  __syncthreads();
  double r = 0;
  if (w == 0) {
    int nw = blockDim.x >> 5;
    r = (l < nw) ? smem[l] : 0.0;
    r = warp_sum(r);
  }
  __syncthreads();
  return r;
}

// The sums of N doubles per thread over the CTA (4 or 8 warps): thread e < N
// returns the sum of value e (0 elsewhere), formed by the trees of block_sum.
// One barrier and N + 3 (N > 1) FP64 additions a warp instead of 2 N barriers
// and 5 N: the FP64 pipe takes 19 cycles of the SM for each, which was a third
// of the back-substitution and a fifth of the mixed cost kernel on 512 windows.
// smem [N * warps].
template <int N>
__device__ double block_sums(double (&v)[N], double* smem) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int base, count;
  warp_scatter_sums<N>(v, lane, base, count);
#pragma unroll
  for (int e = 0; e < warp_scatter_max(N); ++e)
    if (e < count) smem[(base + e) * nw + w] = v[e];
  __syncthreads();
  if (threadIdx.x >= N) return 0.0;
  const double* p = smem + threadIdx.x * nw;
  return nw == 8 ? ((p[0] + p[4]) + (p[2] + p[6])) + ((p[1] + p[5]) + (p[3] + p[7]))
                 : (p[0] + p[2]) + (p[1] + p[3]);
}

// Maxima over the CTA without the FP64 pipe: non-negative numbers are ordered
// as their bits; negative ones and NaN count as 0 (as fmax from 0 does).
__device__ __forceinline__ unsigned long long max_bits(float v) {
  return __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(v, 0.0f)));
}
__device__ __forceinline__ unsigned long long max_bits(double v) {
  const long long b = __double_as_longlong(v);
  unsigned long long m = b > 0 && b <= 0x7ff0000000000000LL ? (unsigned long long)b : 0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long q = __shfl_xor_sync(0xffffffffu, m, o);
    m = q > m ? q : m;
  }
  return m;
}
__device__ __forceinline__ double max_value(unsigned long long bits, float) {
  return double(__uint_as_float(unsigned(bits)));
}
__device__ __forceinline__ double max_value(unsigned long long bits, double) { return bitsd(bits); }
// a and b over the CTA into *ma and *mb (as ordered bits, atomically), smem [2 * warps]
template <typename T>
__device__ void block_max2(T a, T b, unsigned long long* smem, unsigned long long* ma, unsigned long long* mb) {
  const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned long long wa = max_bits(a), wb = max_bits(b);
  if ((threadIdx.x & 31) == 0) {
    smem[w] = wa;
    smem[nw + w] = wb;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long m = 0ull;
    for (int i = 0; i < nw; ++i) {
      const unsigned long long q = smem[threadIdx.x * nw + i];
      m = q > m ? q : m;
    }
    atomicMax(threadIdx.x == 0 ? ma : mb, dbits(max_value(m, T(0))));
  }
}

// Arrival of this CTA at problem p's counter after thread 0 has written the
// CTA's partial sums; true in every thread of the CTA that arrives last of
// `total` (which then runs the problem's LM control step and resets the
// counter for the next launch).  The fence orders this CTA's partials
// before its arrival; the last CTA reads the others' through L2.
__device__ bool last_arrival(unsigned* counter, int total, int* flag_smem) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(counter, 1u);
    const int last = prev == unsigned(total - 1);
    if (last) {
      atomicExch(counter, 0u);
      __threadfence();
    }
    *flag_smem = last;
  }
  __syncthreads();
  return *flag_smem != 0;
}

template <bool CG>
__device__ void ctrl_step_body(const DevPlan& d, int p, double* red);
template <bool CG>
__device__ void ctrl_accept_body(const DevPlan& d, int p, double* red);

// Huber rho and IRLS weight of a squared whitened residual s (Ceres'
// HuberLoss semantics, restated from camera_shared_ceres_optimizor.hpp:253).
__device__ __forceinline__ void loss_eval(int loss, double delta, double s, double& rho, double& w) {
  if (loss == GBA_LOSS_HUBER && s > delta * delta) {
    double r = sqrt(s);
    rho = 2.0 * delta * r - delta * delta;
    w = delta / r;
  } else {
    rho = s;
    w = 1.0;
  }
}

// ---------------------------------------------------------------------------
// Double-float arithmetic: a value is the unevaluated sum hi + lo of two
// floats (about 48 significant bits).  Error-free transformations: Knuth's
// two-sum, Dekker's fast two-sum, and the FMA-based exact product; the
// reciprocal is one Newton step from the float reciprocal.  Used by the
// mixed path to evaluate projections at FP64-class accuracy on the FP32
// pipes (the FP64 pipe of this part issues at 1/57 of the FP32 rate).
// ---------------------------------------------------------------------------
struct ff {
  float hi, lo;
};
__device__ __forceinline__ ff ff_two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ ff ff_fast_two_sum(float a, float b) {
  const float s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ ff ff_add(ff x, ff y) {
  const ff s = ff_two_sum(x.hi, y.hi);
  return ff_fast_two_sum(s.hi, s.lo + (x.lo + y.lo));
}
__device__ __forceinline__ ff ff_add_f(ff x, float y) {
  const ff s = ff_two_sum(x.hi, y);
  return ff_fast_two_sum(s.hi, s.lo + x.lo);
}
__device__ __forceinline__ ff ff_neg(ff x) { return {-x.hi, -x.lo}; }
__device__ __forceinline__ ff ff_mul(ff x, ff y) {
  const float p = x.hi * y.hi;
  float e = fmaf(x.hi, y.hi, -p);
  e = fmaf(x.hi, y.lo, e);
  e = fmaf(x.lo, y.hi, e);
  return ff_fast_two_sum(p, e);
}
__device__ __forceinline__ ff ff_mul_f(ff x, float y) {
  const float p = x.hi * y;
  float e = fmaf(x.hi, y, -p);
  e = fmaf(x.lo, y, e);
  return ff_fast_two_sum(p, e);
}
__device__ __forceinline__ ff ff_fma(ff a, ff b, ff c) { return ff_add(ff_mul(a, b), c); }
__device__ __forceinline__ ff ff_rcp(ff y) {
  const float r = 1.0f / y.hi;
  const ff e = ff_add_f(ff_neg(ff_mul_f(y, r)), 1.0f);   // 1 - y r
  return ff_add_f(ff_mul_f(e, r), r);                    // r + r (1 - y r)
}
__host__ __device__ __forceinline__ float2 ff_split(double d) {
  const float hi = float(d);
  return make_float2(hi, float(d - double(hi)));
}
__device__ __forceinline__ ff ff_ld(float2 v) { return {v.x, v.y}; }

// Rodrigues coefficients of an angle-axis vector.  Near theta = 0 the
// reference formulas divide by zero (analytical_jacobian_matrix_calculator.hpp
// :359-380); series of sin and cos are used below theta = 1e-2.
//   s  = sin(t)/t, c = (1 - cos t)/t^2,
//   a1 = (t cos t - sin t)/t^3, a2 = (t sin t - 2(1 - cos t))/t^4.
__device__ void rodrigues_coeffs(double theta, double& ct, double& s, double& c, double& a1,
                                 double& a2) {
  double t2 = theta * theta;
  if (theta < 1e-2) {
    double t4 = t2 * t2;
    ct = 1.0 - t2 / 2.0 + t4 / 24.0;
    s = 1.0 - t2 / 6.0 + t4 / 120.0;
    c = 0.5 - t2 / 24.0 + t4 / 720.0;
    a1 = -1.0 / 3.0 + t2 / 30.0 - t4 / 840.0;
    a2 = -1.0 / 12.0 + t2 / 180.0 - t4 / 6720.0;
  } else {
    double st;
    sincos(theta, &st, &ct);
    s = st / theta;
    c = (1.0 - ct) / t2;
    a1 = (theta * ct - st) / (t2 * theta);
    a2 = (theta * st - 2.0 * (1.0 - ct)) / (t2 * t2);
  }
}

// ---------------------------------------------------------------------------
// Device projection in FP64 (camera_shared_vector_function.hpp:634-744 with
// radial_distortor.hpp:14-28, decentering_distortor.hpp:14-24).  The camera
// is the full 10-parameter model [k1 k2 k3 d1 d2 f s cx cy a]; groups absent
// from the intrinsic mask hold the identity values (0 / f=1 s=0 c=0 a=1),
// which reproduce the reference's per-mask projection exactly.
// ---------------------------------------------------------------------------
// The FP64 pipe takes 64 cycles an instruction and warp (76 with all four
// schedulers busy), so everything here is written as FMAs, the camera's
// absent terms are left out (their parameters are tested as integers), and
// the Jacobian reuses the projection's terms.
struct Proj64 {
  double w[3];          // R X
  double iz, n0, n1;    // 1 / depth, the undistorted normalized key
  double r2, q;         // n0^2 + n1^2, 1 + radial coefficient
  double e0, e1;        // the distorted normalized key
  double u, v;          // the image key
};

__device__ __forceinline__ bool nonzero64(double x) { return (__double_as_longlong(x) << 1) != 0; }

__device__ __forceinline__ void project64(const double* R, const double* X, const double* cam, Proj64& p) {
#pragma unroll
  for (int m = 0; m < 3; ++m) p.w[m] = fma(R[3 * m + 2], X[2], fma(R[3 * m + 1], X[1], R[3 * m] * X[0]));
  p.iz = 1.0 / (p.w[2] + R[11]);
  p.n0 = (p.w[0] + R[9]) * p.iz;
  p.n1 = (p.w[1] + R[10]) * p.iz;
  p.r2 = fma(p.n1, p.n1, p.n0 * p.n0);
  p.q = 1.0;
  double e0 = p.n0, e1 = p.n1;
  if (nonzero64(cam[0]) || nonzero64(cam[1]) || nonzero64(cam[2])) {
    const double c = p.r2 * fma(p.r2, fma(p.r2, cam[2], cam[1]), cam[0]);
    p.q = __dadd_rn(1.0, c);   // (never contracted: the same bits in every caller)
    e0 = fma(c, e0, e0);
    e1 = fma(c, e1, e1);
  }
  if (nonzero64(cam[3]) || nonzero64(cam[4])) {
    const double x2 = p.n0 + p.n0, xy2 = x2 * p.n1;
    e0 = fma(cam[3], xy2, fma(cam[4], fma(x2, p.n0, p.r2), e0));
    e1 = fma(cam[4], xy2, fma(cam[3], fma(p.n1 + p.n1, p.n1, p.r2), e1));
  }
  p.e0 = e0;
  p.e1 = e1;
  p.u = fma(cam[5], e0, cam[7]);
  if (nonzero64(cam[6])) p.u = fma(cam[6], e1, p.u);
  p.v = fma(cam[5] * cam[9], e1, cam[8]);
}

// The 2x3 point block jp and the 2x6 image block ji of a key from its
// projection.  With M = d(u, v) / d(n0, n1) (distortion and intrinsics) and
// b = M [iz 0 -n0 iz; 0 iz -n1 iz] = d(u, v) / d(camera point): the
// translation columns are b, jp = b R, and as d(R X) / dr = -[R X]x Jl with
// the left Jacobian Jl of the image's angle-axis vector, the rotation columns
// are (R X x b) Jl for each row of b.  These are the derivatives of the
// reference's chain (:334-524) in 70 FP64 instructions instead of about 420.
// l00, l10, l11 and sw whiten and weight M (and so every column); unit false
// when they are the identity.
__device__ __forceinline__ void jacobian64(const double* R, const double* Jl, const double* cam, const Proj64& p,
                                           bool unit, double l00, double l10, double l11, double sw, double* jp,
                                           double* ji) {
  double e00 = p.q, e01 = 0.0, e11 = p.q;
  if (nonzero64(cam[0]) || nonzero64(cam[1]) || nonzero64(cam[2])) {
    const double dc = 2.0 * fma(p.r2, fma(p.r2, 3.0 * cam[2], 2.0 * cam[1]), cam[0]);
    const double t = dc * p.n0;
    e00 = fma(t, p.n0, e00);
    e01 = t * p.n1;
    e11 = fma(dc * p.n1, p.n1, e11);
  }
  if (nonzero64(cam[3]) || nonzero64(cam[4])) {
    const double x1 = 2.0 * cam[3], x2 = 2.0 * cam[4];
    e00 = fma(x1, p.n1, fma(3.0 * x2, p.n0, e00));
    e01 = fma(x1, p.n0, fma(x2, p.n1, e01));
    e11 = fma(x2, p.n0, fma(3.0 * x1, p.n1, e11));
  }
  const double f = cam[5], fa = cam[5] * cam[9];
  double m00 = f * e00, m01 = f * e01, m10 = fa * e01, m11 = fa * e11;
  if (nonzero64(cam[6])) {
    m00 = fma(cam[6], e01, m00);
    m01 = fma(cam[6], e11, m01);
  }
  if (!unit) {
    m00 = sw * fma(l00, m00, l10 * m10);
    m01 = sw * fma(l00, m01, l10 * m11);
    m10 = sw * (l11 * m10);
    m11 = sw * (l11 * m11);
  }
  const double b[2][3] = {{m00 * p.iz, m01 * p.iz, 0.0}, {m10 * p.iz, m11 * p.iz, 0.0}};
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const double b0 = b[r][0], b1 = b[r][1], b2 = -fma(b0, p.n0, b1 * p.n1);
    const double c0 = fma(p.w[1], b2, -(p.w[2] * b1)), c1 = fma(p.w[2], b0, -(p.w[0] * b2)),
                 c2 = fma(p.w[0], b1, -(p.w[1] * b0));
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      jp[3 * r + j] = fma(b2, R[6 + j], fma(b1, R[3 + j], b0 * R[j]));
      ji[6 * r + j] = fma(c2, Jl[6 + j], fma(c1, Jl[3 + j], c0 * Jl[j]));
    }
    ji[6 * r + 3] = b0;
    ji[6 * r + 4] = b1;
    ji[6 * r + 5] = b2;
  }
}

// Analytical Jacobian of one key in precision T: jp 2x3, ji 2x6 (row-major).
// IL = [r0 r1 r2 t0 t1 t2 ct s c a1 a2 pad] of the image.  Follows
// WorldPointToNormalizedPointDerivation (:334-429), RadialDistortDerivation
// (:431-470), DecenteringDistortDerivation (:472-503) and the intrinsic
// chains (:505-524).
template <typename T>
__device__ __forceinline__ void key_jacobian(const T* X, const T* IL, const T* cam, T* jp, T* ji,
                                             T* nrm = nullptr) {
  const T r0 = IL[0], r1 = IL[1], r2 = IL[2];
  const T ct = IL[6], s = IL[7], c = IL[8], a1 = IL[9], a2 = IL[10];
  const T d = r0 * X[0] + r1 * X[1] + r2 * X[2];
  const T v0 = r1 * X[2] - r2 * X[1], v1 = r2 * X[0] - r0 * X[2], v2 = r0 * X[1] - r1 * X[0];
  const T y0 = ct * X[0] + s * v0 + c * d * r0 + IL[3];
  const T y1 = ct * X[1] + s * v1 + c * d * r1 + IL[4];
  const T y2 = ct * X[2] + s * v2 + c * d * r2 + IL[5];
  // pypr = w r^T + s [pvpr] + c (d I + r X^T),  w = -s X + a1 v + a2 d r
  const T w0 = -s * X[0] + a1 * v0 + a2 * d * r0;
  const T w1 = -s * X[1] + a1 * v1 + a2 * d * r1;
  const T w2 = -s * X[2] + a1 * v2 + a2 * d * r2;
  T pr[3][3];
  pr[0][0] = w0 * r0 + c * (d + r0 * X[0]);
  pr[0][1] = w0 * r1 + s * X[2] + c * r0 * X[1];
  pr[0][2] = w0 * r2 - s * X[1] + c * r0 * X[2];
  pr[1][0] = w1 * r0 - s * X[2] + c * r1 * X[0];
  pr[1][1] = w1 * r1 + c * (d + r1 * X[1]);
  pr[1][2] = w1 * r2 + s * X[0] + c * r1 * X[2];
  pr[2][0] = w2 * r0 + s * X[1] + c * r2 * X[0];
  pr[2][1] = w2 * r1 - s * X[0] + c * r2 * X[1];
  pr[2][2] = w2 * r2 + c * (d + r2 * X[2]);
  // pypp = ct I + s [r]x + c r r^T
  T pp[3][3];
  pp[0][0] = ct + c * r0 * r0; pp[0][1] = -s * r2 + c * r0 * r1; pp[0][2] = s * r1 + c * r0 * r2;
  pp[1][0] = s * r2 + c * r1 * r0; pp[1][1] = ct + c * r1 * r1; pp[1][2] = -s * r0 + c * r1 * r2;
  pp[2][0] = -s * r1 + c * r2 * r0; pp[2][1] = s * r0 + c * r2 * r1; pp[2][2] = ct + c * r2 * r2;
  const T iz = T(1) / y2;
  const T n0 = y0 * iz, n1 = y1 * iz;
  if (nrm) {
    nrm[0] = n0;
    nrm[1] = n1;
  }
  // normalized-key derivatives A (2 x 9): columns 0..2 point, 3..8 image
  T A0[9], A1[9];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    A0[m] = (pp[0][m] - n0 * pp[2][m]) * iz;
    A1[m] = (pp[1][m] - n1 * pp[2][m]) * iz;
    A0[3 + m] = (pr[0][m] - n0 * pr[2][m]) * iz;
    A1[3 + m] = (pr[1][m] - n1 * pr[2][m]) * iz;
  }
  A0[6] = iz; A0[7] = T(0); A0[8] = -n0 * iz;
  A1[6] = T(0); A1[7] = iz; A1[8] = -n1 * iz;
  // distortion chains (both from the undistorted key and A)
  const T rr2 = n0 * n0 + n1 * n1, rr4 = rr2 * rr2;
  const T coeff = cam[0] * rr2 + cam[1] * rr4 + cam[2] * rr4 * rr2;
  const T dcoef = cam[0] + T(2) * cam[1] * rr2 + T(3) * cam[2] * rr4;
  const T d1 = cam[3], d2 = cam[4];
  const T f = cam[5], sk = cam[6], fa = cam[5] * cam[9];
  // (a camera without distortion adds zeros only: left out, the same values)
  T e0[9], e1[9];
  if (cam[0] != T(0) || cam[1] != T(0) || cam[2] != T(0) || d1 != T(0) || d2 != T(0)) {
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      const T pr2 = T(2) * (n0 * A0[j] + n1 * A1[j]);
      const T cd = dcoef * pr2;
      const T cross = A0[j] * n1 + A1[j] * n0;
      e0[j] = A0[j] + (cd * n0 + coeff * A0[j]) + (T(2) * d1 * cross + d2 * (pr2 + T(4) * n0 * A0[j]));
      e1[j] = A1[j] + (cd * n1 + coeff * A1[j]) + (T(2) * d2 * cross + d1 * (pr2 + T(4) * n1 * A1[j]));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 9; ++j) {
      e0[j] = A0[j];
      e1[j] = A1[j];
    }
  }
  T out0[9], out1[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    out0[j] = f * e0[j] + sk * e1[j];
    out1[j] = fa * e1[j];
  }
#pragma unroll
  for (int m = 0; m < 3; ++m) { jp[m] = out0[m]; jp[3 + m] = out1[m]; }
#pragma unroll
  for (int m = 0; m < 6; ++m) { ji[m] = out0[3 + m]; ji[6 + m] = out1[3 + m]; }
}

template <typename T>
__device__ __forceinline__ const T* tptr(const void* p) { return static_cast<const T*>(p); }
template <typename T>
__device__ __forceinline__ T* tptr_mut(void* p) { return static_cast<T*>(p); }

template <typename T>
__device__ __forceinline__ void load_cam(const DevPlan& d, int par, int cam, T* out);
template <>
__device__ __forceinline__ void load_cam<float>(const DevPlan& d, int par, int cam, float* out) {
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(d.cam32[par] + 10LL * cam) + j);
    out[2 * j] = v.x;
    out[2 * j + 1] = v.y;
  }
}
template <>
__device__ __forceinline__ void load_cam<double>(const DevPlan& d, int par, int cam, double* out) {
#pragma unroll
  for (int j = 0; j < 10; ++j) out[j] = d.cam64[par][10 * cam + j];
}

// Derivatives of the image key with respect to all ten camera parameters in
// the full model's order [k1 k2 k3][d1 d2][f s cx cy a]
// (camera_shared_analytical_jacobian_matrix_calculator.hpp:526-557), from the
// undistorted normalized key n: row 0 (u) in jc[0..9], row 1 (v) in
// jc[10..19].  Consumers pick the computed parameters' columns.
template <typename T>
__device__ __forceinline__ void camera_jacobian(T n0, T n1, const T* cam, T* jc) {
  const T r2 = n0 * n0 + n1 * n1, r4 = r2 * r2, r6 = r4 * r2;
  const T coeff = cam[0] * r2 + cam[1] * r4 + cam[2] * r6;
  const T d1 = cam[3], d2 = cam[4];
  const T e0 = n0 + coeff * n0 + (T(2) * d1 * n0 * n1 + d2 * (r2 + T(2) * n0 * n0));
  const T e1 = n1 + coeff * n1 + (T(2) * d2 * n0 * n1 + d1 * (r2 + T(2) * n1 * n1));
  const T f = cam[5], sk = cam[6], a = cam[9];
  // distortion columns through K: u = f e0 + s e1 + cx, v = f a e1 + cy
  const T de0[5] = {r2 * n0, r4 * n0, r6 * n0, T(2) * n0 * n1, r2 + T(2) * n0 * n0};
  const T de1[5] = {r2 * n1, r4 * n1, r6 * n1, r2 + T(2) * n1 * n1, T(2) * n0 * n1};
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    jc[m] = f * de0[m] + sk * de1[m];
    jc[10 + m] = f * a * de1[m];
  }
  jc[5] = e0;    jc[15] = a * e1;   // f
  jc[6] = e1;    jc[16] = T(0);     // s
  jc[7] = T(1);  jc[17] = T(0);     // cx
  jc[8] = T(0);  jc[18] = T(1);     // cy
  jc[9] = T(0);  jc[19] = f * e1;   // a
}

// The same in FP64 from the key's projection (every rounding explicit, so the
// bits do not depend on the calling kernel).
__device__ __forceinline__ void camera_jacobian64(const Proj64& p, const double* cam, double* jc) {
  const double r4 = p.r2 * p.r2, r6 = r4 * p.r2, x2 = p.n0 + p.n0, xy2 = x2 * p.n1;
  const double f = cam[5], sk = cam[6], a = cam[9], fa = f * a;
  const double de0[5] = {p.r2 * p.n0, r4 * p.n0, r6 * p.n0, xy2, fma(x2, p.n0, p.r2)};
  const double de1[5] = {p.r2 * p.n1, r4 * p.n1, r6 * p.n1, fma(p.n1 + p.n1, p.n1, p.r2), xy2};
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    jc[m] = fma(sk, de1[m], f * de0[m]);
    jc[10 + m] = fa * de1[m];
  }
  jc[5] = p.e0;  jc[15] = a * p.e1;   // f
  jc[6] = p.e1;  jc[16] = 0.0;        // s
  jc[7] = 1.0;   jc[17] = 0.0;        // cx
  jc[8] = 0.0;   jc[18] = 1.0;        // cy
  jc[9] = 0.0;   jc[19] = f * p.e1;   // a
}

// Column of the full ten [k1 k2 k3 d1 d2 f s cx cy a] holding a camera's
// computed parameter m, or -1 past its count.
__host__ __device__ __forceinline__ int cam_full_col(unsigned mask, int m) {
  if (mask & GBA_COMPUTE_RADIAL_DISTORTION) {
    if (m < 3) return m;
    m -= 3;
  }
  if (mask & GBA_COMPUTE_DECENTERING_DISTORTION) {
    if (m < 2) return 3 + m;
    m -= 2;
  }
  if ((mask & GBA_COMPUTE_INTRINSIC_PARAMS) && m < 5) return 5 + m;
  return -1;
}

// The computed parameter held in full column j, or -1 when j is not computed.
__device__ __forceinline__ int cam_compact_col(unsigned mask, int j) {
  const int nr = (mask & GBA_COMPUTE_RADIAL_DISTORTION) ? 3 : 0;
  const int nd = (mask & GBA_COMPUTE_DECENTERING_DISTORTION) ? 2 : 0;
  if (j < 3) return nr ? j : -1;
  if (j < 5) return nd ? nr + j - 3 : -1;
  return (mask & GBA_COMPUTE_INTRINSIC_PARAMS) ? nr + nd + j - 5 : -1;
}

// Index of (a, b), a <= b, in the row-major upper triangle of a 10 x 10 block.
__device__ __forceinline__ int upper10(int a, int b) { return 10 * a - a * (a - 1) / 2 + (b - a); }


// ---------------------------------------------------------------------------
// init / copy x0
// ---------------------------------------------------------------------------
__global__ void k_init(DevPlan d) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < d.B) {
    LMState st = {};
    st.nu = 2.0;
    st.active = 1;
    st.relin = 1;
    st.first = 1;
    st.factor_ok = 1;
    st.stop = GBA_STOP_MAX_ITERATIONS;
    st.status = GBA_OK;
    st.loop_total = d.state[p].loop_total;   // (of the plan, not of this run)
    d.state[p] = st;
    d.factor_flag[p] = 0;
  }
}

__global__ void k_copy_x0(DevPlan d) {
  long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  long long np = 3LL * d.P, ni = 6LL * d.I, nc = d.free_cams ? 10LL * d.Ctot : 0;
  if (i < np) {
    d.x_pt[0][i] = d.x0_pt[i];
    if (d.x_ff[0]) d.x_ff[0][i] = ff_split(d.x0_pt[i]);
  } else if (i < np + ni) {
    d.x_img[0][i - np] = d.x0_img[i - np];
  } else if (i < np + ni + nc) {
    d.x_cam[0][i - np - ni] = d.x0_cam[i - np - ni];
  }
}

// Free cameras: the ten-parameter camera of x_cam (which = 0 current, 1
// candidate) in every form the key kernels read.  Fixed cameras keep the
// values uploaded at plan creation in both parities.
__global__ void k_cam_prep(DevPlan d, int which) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.Ctot) return;
  const int4 ci = d.cam_info[c];
  if (ci.x == 0) return;
  const LMState& st = d.state[ci.z];
  if (which == 0 ? !st.active : !st.evaluate) return;
  const int par = which ? 1 - st.parity : st.parity;
  const double* x = d.x_cam[par] + 10LL * c;
  double full[10] = {0, 0, 0, 0, 0, 1, 0, 0, 0, 1};
#pragma unroll
  for (int j = 0; j < 10; ++j) {
    const int m = cam_compact_col(unsigned(ci.y), j);
    if (m >= 0) full[j] = x[m];
  }
#pragma unroll
  for (int j = 0; j < 10; ++j) {
    d.cam64[par][10LL * c + j] = full[j];
    d.cam32[par][10LL * c + j] = float(full[j]);
  }
  if (d.cam_ff[par]) {
#pragma unroll
    for (int j = 0; j < 9; ++j) d.cam_ff[par][10LL * c + j] = ff_split(full[j]);
    d.cam_ff[par][10LL * c + 9] = ff_split(full[5] * full[9]);   // f * a
  }
}

// ---------------------------------------------------------------------------
// image prep: which = 0 current x (at init), 1 candidate x (when evaluating)
// ---------------------------------------------------------------------------
// The rotation of image i's parameters in parity par in every form the key
// kernels read.
template <typename T>
__device__ void image_prep_one(const DevPlan& d, int i, int par) {
  const double* x = d.x_img[par] + 6LL * i;
  double r0 = x[0], r1 = x[1], r2 = x[2];
  double theta = sqrt(r0 * r0 + r1 * r1 + r2 * r2);
  double ct, s, c, a1, a2;
  rodrigues_coeffs(theta, ct, s, c, a1, a2);
  double* R = d.img_rot[par] + 12LL * i;
  if (theta == 0.0) {  // :695-698 -- camera point = X + t
    R[0] = 1; R[1] = 0; R[2] = 0; R[3] = 0; R[4] = 1; R[5] = 0; R[6] = 0; R[7] = 0; R[8] = 1;
  } else {
    // R = cos I + sin [k]x + (1 - cos) k k^T, k = r / theta
    double st_ = s * theta, omc = c * theta * theta;
    double k0 = r0 / theta, k1 = r1 / theta, k2 = r2 / theta;
    R[0] = ct + omc * k0 * k0; R[1] = -st_ * k2 + omc * k0 * k1; R[2] = st_ * k1 + omc * k0 * k2;
    R[3] = st_ * k2 + omc * k1 * k0; R[4] = ct + omc * k1 * k1; R[5] = -st_ * k0 + omc * k1 * k2;
    R[6] = -st_ * k1 + omc * k2 * k0; R[7] = st_ * k0 + omc * k2 * k1; R[8] = ct + omc * k2 * k2;
  }
  R[9] = x[3]; R[10] = x[4]; R[11] = x[5];
  if (d.img_rot_ff[par]) {
    float2* Rf = d.img_rot_ff[par] + 12LL * i;
#pragma unroll
    for (int j = 0; j < 12; ++j) Rf[j] = ff_split(R[j]);
  }
  T* IL = tptr_mut<T>(d.img_lin[par]) + 12LL * i;
  if constexpr (sizeof(T) == sizeof(double)) {
    // left Jacobian of the angle-axis vector: s I + c [r]x + b r r^T, b =
    // (1 - s) / theta^2 (jacobian64; its rows, then padding)
    const double t2 = theta * theta;
    const double b = theta < 1e-2 ? 1.0 / 6.0 - t2 / 120.0 + t2 * t2 / 5040.0 : (1.0 - s) / t2;
    IL[0] = s + b * r0 * r0;       IL[1] = b * r0 * r1 - c * r2;  IL[2] = b * r0 * r2 + c * r1;
    IL[3] = b * r1 * r0 + c * r2;  IL[4] = s + b * r1 * r1;       IL[5] = b * r1 * r2 - c * r0;
    IL[6] = b * r2 * r0 - c * r1;  IL[7] = b * r2 * r1 + c * r0;  IL[8] = s + b * r2 * r2;
    IL[9] = IL[10] = IL[11] = 0.0;
  } else {
    IL[0] = T(r0); IL[1] = T(r1); IL[2] = T(r2);
    IL[3] = T(x[3]); IL[4] = T(x[4]); IL[5] = T(x[5]);
    IL[6] = T(ct); IL[7] = T(s); IL[8] = T(c); IL[9] = T(a1); IL[10] = T(a2); IL[11] = T(0);
  }
}

// which = 0: the current x of active problems (at init); 1: the candidate of
// problems whose step is evaluated.  The solve loop prepares the candidate in
// k_backsub instead; which = 1 is kept for callers that move x themselves.
template <typename T>
__global__ void k_image_prep(DevPlan d, int which) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.I) return;
  const LMState& st = d.state[d.img_prob[i]];
  if (which == 0 ? !st.active : !st.evaluate) return;
  image_prep_one<T>(d, i, which ? 1 - st.parity : st.parity);
}

// Soft-constraint and point-prior part of the cost, sum w (x - y)^2 and
// (x - y)^T L (x - y) (no loss), one CTA per problem over its rows
// (camera_shared_mahalanobis_distance_calculator.hpp:28-58).
__global__ void __launch_bounds__(256) k_cons_cost(DevPlan d, int which) {
  __shared__ double red[32];
  const int p = blockIdx.x;
  const LMState& st = d.state[p];
  if (which == 0 ? !st.active : !st.evaluate) return;
  const int par = which ? 1 - st.parity : st.parity;
  double acc = 0.0;
  if (d.n_cons > 0)
    for (int r = d.prob_cons_off[p] + threadIdx.x; r < d.prob_cons_off[p + 1]; r += blockDim.x) {
      const int4 c = d.cons[r];
      const double2 yw = d.cons_yw[r];
      const double x = c.x == 0   ? d.x_pt[par][3LL * c.y + c.z]
                       : c.x == 1 ? d.x_img[par][6LL * c.y + c.z]
                                  : d.x_cam[par][10LL * c.y + c.z];
      const double v = x - yw.x;
      acc += yw.y * v * v;
    }
  if (d.n_priors > 0)   // (x - y)^T L (x - y) per prior (ba_gcp_constrained_mahalanobis_distance_calculator.hpp:55-62)
    for (int i = d.prob_prior_off[p] + threadIdx.x; i < d.prob_prior_off[p + 1]; i += blockDim.x) {
      const double* xp = d.x_pt[par] + 3LL * d.prior_pt[i];
      const double* L = d.prior_info + 9LL * i;
      double v[3];
      for (int a = 0; a < 3; ++a) v[a] = xp[a] - d.prior_y[3LL * i + a];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) acc += v[a] * L[3 * a + b] * v[b];
    }
  acc = block_sum(acc, red);
  if (threadIdx.x == 0) d.cons_cost[p] = acc;
}

// ---------------------------------------------------------------------------
// cost: FP64 residual per key, whitened and weighted residual stored in T
// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// linearize, one thread per key (coalesced JR records): the analytical
// Jacobian of the key, whitened by the key weight and the IRLS weight, into
// the records of parity `par` (and the camera block with free cameras).
// X, il, cam are the point, the image's linearisation coefficients and the
// camera at that parity; rw0, rw1, sw the key's weighted residual and the
// square root of its IRLS weight.
// ---------------------------------------------------------------------------
// The camera block jc of key k (free cameras), whitened and weighted as the
// others, into JC.
__device__ __forceinline__ float whiten_u(float l00, float a, float l10, float b) { return l00 * a + l10 * b; }
__device__ __forceinline__ double whiten_u(double l00, double a, double l10, double b) { return fma(l00, a, l10 * b); }

// FP32 records (80 bytes: five 16-byte words) of a warp's keys on their way to
// memory: each lane puts its own into its slot, and the warp writes the slots
// word by word to consecutive addresses, whole sectors.  A record to a lane,
// every store instruction left 32 half-written sectors 80 bytes apart (the
// free-camera grid with its two records a key: 70 -> 61 us).  The odd pitch
// keeps both sides free of bank conflicts.  Reading records this way was
// slower (point sums of 512 windows 477 -> 610 us): L1 holds the lines between
// a lane's five loads, and shared memory and registers cost warps.
constexpr int kRecWords = kJRStride * int(sizeof(float)) / 16;
using RecordSlots = uint4[32 * kRecWords];

// The first n slots to the records of keys k, k + 1, ...
__device__ __forceinline__ void store_record_slots(float* recs, long long k, int n, const RecordSlots& slots, int lane) {
  uint4* w = reinterpret_cast<uint4*>(recs) + kRecWords * k;
  __syncwarp();
#pragma unroll
  for (int u = 0; u < kRecWords; ++u) {
    const int c = lane + 32 * u;
    if (c < kRecWords * n) w[c] = slots[c];
  }
  __syncwarp();
}

template <typename T>
__device__ __forceinline__ void linearize_cam(const DevPlan& d, int k, T* jc, T sw, T* out) {
  T l00 = T(1), l10 = T(0), l11 = T(1);
  if (d.key_wl) {
    l00 = T(__ldg(d.key_wl + 3LL * k));
    l10 = T(__ldg(d.key_wl + 3LL * k + 1));
    l11 = T(__ldg(d.key_wl + 3LL * k + 2));
  }
#pragma unroll
  for (int m = 0; m < 10; ++m) {
    const T a = jc[m], b = jc[10 + m];
    jc[m] = whiten_u(l00, a, l10, b) * sw;
    jc[10 + m] = l11 * b * sw;
  }
  store_vec<20>(out, jc);
}

// The FP32 records of a warp's keys k0 .. k0 + n - 1 (this lane's: k).
__device__ __forceinline__ void linearize_key(const DevPlan& d, int k, int par, int fix, const float* X,
                                              const float* il, const float* cam, float rw0, float rw1, float sw,
                                              RecordSlots& slots, int lane, int k0, int n) {
  float* const own = reinterpret_cast<float*>(slots + lane * kRecWords);
  float jp[6], ji[12], nrm[2];
  key_jacobian<float>(X, il, cam, jp, ji, nrm);
  if (fix & 1) {   // fixed points: no point columns
#pragma unroll
    for (int m = 0; m < 6; ++m) jp[m] = 0.0f;
  }
  if (fix & 2) {   // fixed images: no image columns
#pragma unroll
    for (int m = 0; m < 12; ++m) ji[m] = 0.0f;
  }
  if (d.free_cams) {
    float jc[20];
    camera_jacobian<float>(nrm[0], nrm[1], cam, jc);
    linearize_cam<float>(d, k, jc, sw, own);
    store_record_slots(tptr_mut<float>(d.JC[par]), k0, n, slots, lane);   // (20 values too)
  }
  if (d.key_wl) {
    const float l00 = float(__ldg(d.key_wl + 3LL * k)), l10 = float(__ldg(d.key_wl + 3LL * k + 1)),
                l11 = float(__ldg(d.key_wl + 3LL * k + 2));
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const float a = jp[m], b = jp[3 + m];
      jp[m] = (l00 * a + l10 * b) * sw;
      jp[3 + m] = l11 * b * sw;
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const float a = ji[m], b = ji[6 + m];
      ji[m] = (l00 * a + l10 * b) * sw;
      ji[6 + m] = l11 * b * sw;
    }
  } else {
#pragma unroll
    for (int m = 0; m < 6; ++m) jp[m] *= sw;
#pragma unroll
    for (int m = 0; m < 12; ++m) ji[m] *= sw;
  }
  float rec[kJRStride];
#pragma unroll
  for (int m = 0; m < 6; ++m) rec[m] = jp[m];
#pragma unroll
  for (int m = 0; m < 12; ++m) rec[6 + m] = ji[m];
  rec[18] = rw0;
  rec[19] = rw1;
  store_vec<kJRStride>(own, rec);
  store_record_slots(tptr_mut<float>(d.JR[par]), k0, n, slots, lane);
}

// The FP64 record of key k from its projection p and the rotation R of its image.
__device__ __forceinline__ void linearize_key64(const DevPlan& d, int k, int img, int par, int fix, const double* R,
                                                const double* cam, const Proj64& p, double rw0, double rw1,
                                                double sw) {
  double Jl[10], rec[kJRStride];
  load_vec<10>(tptr<double>(d.img_lin[par]) + 12LL * img, Jl);
  double l00 = 1.0, l10 = 0.0, l11 = 1.0;
  if (d.key_wl) {
    l00 = __ldg(d.key_wl + 3LL * k);
    l10 = __ldg(d.key_wl + 3LL * k + 1);
    l11 = __ldg(d.key_wl + 3LL * k + 2);
  }
  const bool unit = !d.key_wl && __double_as_longlong(sw) == __double_as_longlong(1.0);
  jacobian64(R, Jl, cam, p, unit, l00, l10, l11, sw, rec, rec + 6);
  if (fix & 1) {   // fixed points: no point columns
#pragma unroll
    for (int m = 0; m < 6; ++m) rec[m] = 0.0;
  }
  if (fix & 2) {   // fixed images: no image columns
#pragma unroll
    for (int m = 6; m < 18; ++m) rec[m] = 0.0;
  }
  if (d.free_cams) {
    double jc[20];
    camera_jacobian64(p, cam, jc);
    linearize_cam<double>(d, k, jc, sw, tptr_mut<double>(d.JC[par]) + 20LL * k);
  }
  rec[18] = rw0;
  rec[19] = rw1;
  store_vec<kJRStride>(tptr_mut<double>(d.JR[par]) + (long long)kJRStride * k, rec);
}

// The records of a key chunk at parity par, one key per thread.  rws: the
// weighted residuals of the chunk's keys, each written by its own thread, or
// null: from RW.
template <typename T>
__device__ __forceinline__ void linearize_chunk(const DevPlan& d, const Chunk& ch, int par,
                                                const float4* rws = nullptr) {
  const double* __restrict__ xp = d.x_pt[par];
  const T* __restrict__ rwb = tptr<T>(d.RW[par]);
  const int fix = d.prob[ch.prob].fix;
  if constexpr (sizeof(T) == sizeof(float)) {
    __shared__ RecordSlots recs[256 / 32];   // (launched with 256 threads)
    const int lane = threadIdx.x & 31;
    __syncwarp();   // (rws)
    for (int k0 = ch.begin + int(threadIdx.x) - lane; k0 < ch.end; k0 += blockDim.x) {
      const int k = min(k0 + lane, ch.end - 1);   // (the last key again where there is none)
      const int img = __ldg(d.key_img + k), pt = __ldg(d.key_pt + k);
      float cam[10], rw[4], X[3], il[12];
      load_cam<float>(d, par, __ldg(d.img_cam + img), cam);
      if (rws) {
        const float4 v = rws[k - ch.begin];
        rw[0] = v.x; rw[1] = v.y; rw[2] = v.z;
      } else {   // (k_cost_ff has just written them: not through the read-only path)
        const float4 v = __ldcg(reinterpret_cast<const float4*>(rwb + 4LL * k));
        rw[0] = v.x; rw[1] = v.y; rw[2] = v.z;
      }
      if (d.x_ff[par]) {   // mixed: high part of the mirror
        const float2* xf = d.x_ff[par] + 3LL * pt;
        X[0] = xf[0].x; X[1] = xf[1].x; X[2] = xf[2].x;
      } else {
        X[0] = float(xp[3LL * pt]); X[1] = float(xp[3LL * pt + 1]); X[2] = float(xp[3LL * pt + 2]);
      }
      load_vec<12>(tptr<float>(d.img_lin[par]) + 12LL * img, il);
      linearize_key(d, k, par, fix, X, il, cam, rw[0], rw[1], rw[2], recs[threadIdx.x >> 5], lane, k0,
                    min(32, ch.end - k0));
    }
  } else {
    for (int k = ch.begin + threadIdx.x; k < ch.end; k += blockDim.x) {
      const int img = __ldg(d.key_img + k), pt = __ldg(d.key_pt + k);
      T cam[10];
      load_cam<T>(d, par, __ldg(d.img_cam + img), cam);
      T rw[4];
      load_vec<4>(rwb + 4LL * k, rw);
      double R[12];
      load_vec<12>(d.img_rot[par] + 12LL * img, R);
      const double X[3] = {xp[3LL * pt], xp[3LL * pt + 1], xp[3LL * pt + 2]};
      Proj64 p;
      project64(R, X, cam, p);
      linearize_key64(d, k, img, par, fix, R, cam, p, rw[0], rw[1], rw[2]);
    }
  }
}

// The prologue's linearization (and, with DevPlan::fuse_lin off, every
// iteration's): the records at the problem's current parity.
template <typename T>
__global__ void __launch_bounds__(256) k_linearize_keys(DevPlan d) {
  const Chunk ch = d.key_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (!st.relin || !st.active) return;
  linearize_chunk<T>(d, ch, st.parity);
}

// FP64 cost, and for a candidate its Jacobian records from the same
// projection (each key's residual goes into its record; RW is written only
// for a separate linearization).  Bound by the FP64 pipe: about 115
// instructions a key (480 with the chain kept apart for each column: 24
// windows of 0.95 M keys in all 27.6 -> 22.7 ms a solve, grid 4.57 -> 4.0 ms
// an iteration).
__global__ void __launch_bounds__(256) k_cost(DevPlan d, int which) {
  __shared__ double red[32];
  const Chunk ch = d.key_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (which == 0 ? !st.active : !st.evaluate) return;
  const int par = which ? 1 - st.parity : st.parity;
  const bool records = which == 1 && d.fuse_lin;
  const int fix = d.prob[ch.prob].fix;
  const double* __restrict__ xp = d.x_pt[par];
  double* __restrict__ rw = tptr_mut<double>(d.RW[par]);
  double acc = 0.0, acc_raw = 0.0;
  for (int k = ch.begin + threadIdx.x; k < ch.end; k += blockDim.x) {
    const int img = __ldg(d.key_img + k), pt = __ldg(d.key_pt + k);
    double R[12], cam[10];
    // (written by an earlier launch: read-only here)
    load_vec<12>(d.img_rot[par] + 12LL * img, R);
    const double X[3] = {xp[3LL * pt], xp[3LL * pt + 1], xp[3LL * pt + 2]};
    load_vec<10>(d.cam64[par] + 10LL * __ldg(d.img_cam + img), cam);
    Proj64 p;
    project64(R, X, cam, p);
    const double2 ob = __ldg(d.key_obs + k);
    double e0 = p.u - ob.x, e1 = p.v - ob.y;   // r = f(x) - y
    double sq = fma(e1, e1, e0 * e0);
    acc_raw += sq;
    if (d.key_wl) {
      const double l00 = __ldg(d.key_wl + 3LL * k), l10 = __ldg(d.key_wl + 3LL * k + 1),
                   l11 = __ldg(d.key_wl + 3LL * k + 2);
      e0 = fma(l00, e0, l10 * e1);
      e1 = l11 * e1;
      sq = fma(e1, e1, e0 * e0);
    }
    double rho = sq, w, sw = 1.0;
    if (d.loss != GBA_LOSS_TRIVIAL) {
      loss_eval(d.loss, d.huber_delta, sq, rho, w);
      if (w != 1.0) {
        sw = sqrt(w);
        e0 *= sw;
        e1 *= sw;
      }
    }
    acc += rho;
    if (records) {   // the candidate's Jacobian records, used if it is accepted
      linearize_key64(d, k, img, par, fix, R, cam, p, e0, e1, sw);
    } else {
      const double out[4] = {e0, e1, sw, 0.0};
      store_vec<4>(rw + 4LL * k, out);
    }
  }
  double sums[2] = {acc, acc_raw};
  const double tot = block_sums<2>(sums, red);
  if (threadIdx.x < 2) d.key_chunk_sum[2LL * blockIdx.x + threadIdx.x] = tot;
  if (which == 1 && d.fold_ctrl) {   // the accept decision in the last CTA of the problem
    __shared__ int last;
    const int p = ch.prob;
    if (last_arrival(d.fold_count + 2 * p + 1,
                     d.prob_key_chunk_off[p + 1] - d.prob_key_chunk_off[p], &last))
      ctrl_accept_body<true>(d, p, red);
  }
}

// Mixed-path cost: the projection in double-float from the double-float
// mirrors of x, R|t, the keys and the cameras; per-thread sums in
// double-float, block sums in FP64.  Bound by its instructions and by L1 (55%
// and 71% busy, 32 warps an SM): the keys of a warp see many images, so every
// load instruction of an image's values is some 20 lines.  R|t, the camera and
// the key come in 16-byte loads (half as many), which with the records' store
// (store_record_slots) took 512 windows from 1117 to 1012 us, the random walk
// from 485 to 420, the grid from 60.6 to 53.0 and its free cameras from 76 to
// 61.  Without the bound of 64 registers: 80, three blocks an SM, 1249 us.
__global__ void __launch_bounds__(256, 4) k_cost_ff(DevPlan d, int which) {
  __shared__ double red[32];
  __shared__ float4 rws[kKeyChunk];   // the residuals on their way into the records
  const Chunk ch = d.key_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (which == 0 ? !st.active : !st.evaluate) return;
  const int par = which ? 1 - st.parity : st.parity;
  const float2* __restrict__ xp = d.x_ff[par];
  const float2* __restrict__ rot = d.img_rot_ff[par];
  float* __restrict__ rw = static_cast<float*>(d.RW[par]);
  const bool records = which == 1 && d.fuse_lin, local = records && ch.end - ch.begin <= kKeyChunk;
  ff acc = {0.0f, 0.0f};
  double acc_raw = 0.0;
  for (int k = ch.begin + threadIdx.x; k < ch.end; k += blockDim.x) {
    const int img = __ldg(d.key_img + k), pt = __ldg(d.key_pt + k);
    float R[24];
    load_vec<24>(reinterpret_cast<const float*>(rot + 12LL * img), R);
    auto Rm = [&](int m) { return ff{R[2 * m], R[2 * m + 1]}; };
    const ff X0 = ff_ld(xp[3LL * pt]), X1 = ff_ld(xp[3LL * pt + 1]), X2 = ff_ld(xp[3LL * pt + 2]);
    ff y[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      ff a = Rm(9 + m);
      a = ff_fma(Rm(3 * m), X0, a);
      a = ff_fma(Rm(3 * m + 1), X1, a);
      y[m] = ff_fma(Rm(3 * m + 2), X2, a);
    }
    const ff iz = ff_rcp(y[2]);
    ff n0 = ff_mul(y[0], iz), n1 = ff_mul(y[1], iz);
    const float4* cam = reinterpret_cast<const float4*>(d.cam_ff[par] + 10 * __ldg(d.img_cam + img));
    const float4 cam01 = __ldg(cam), cam23 = __ldg(cam + 1), cam45 = __ldg(cam + 2);
    const ff k1 = {cam01.x, cam01.y}, k2 = {cam01.z, cam01.w}, k3 = {cam23.x, cam23.y};
    const ff d1 = {cam23.z, cam23.w}, d2 = {cam45.x, cam45.y};
    const ff r2 = ff_add(ff_mul(n0, n0), ff_mul(n1, n1));
    ff dx = {0.0f, 0.0f}, dy = {0.0f, 0.0f};
    if (k1.hi != 0.0f || k2.hi != 0.0f || k3.hi != 0.0f) {
      const ff coeff = ff_mul(r2, ff_fma(r2, ff_fma(r2, k3, k2), k1));
      dx = ff_mul(coeff, n0);
      dy = ff_mul(coeff, n1);
    }
    if (d1.hi != 0.0f || d2.hi != 0.0f) {
      const ff xy2 = ff_mul_f(ff_mul(n0, n1), 2.0f);
      dx = ff_add(dx, ff_add(ff_mul(d1, xy2), ff_mul(d2, ff_add(r2, ff_mul_f(ff_mul(n0, n0), 2.0f)))));
      dy = ff_add(dy, ff_add(ff_mul(d2, xy2), ff_mul(d1, ff_add(r2, ff_mul_f(ff_mul(n1, n1), 2.0f)))));
    }
    n0 = ff_add(n0, dx);
    n1 = ff_add(n1, dy);
    const float4 cam67 = __ldg(cam + 3), cam89 = __ldg(cam + 4);
    const ff f = {cam45.z, cam45.w}, sk = {cam67.x, cam67.y}, cx = {cam67.z, cam67.w}, cy = {cam89.x, cam89.y};
    const ff fa = {cam89.z, cam89.w};   // f * a, stored pre-multiplied
    const ff u = ff_add(ff_fma(f, n0, ff_mul(sk, n1)), cx);
    const ff v = ff_fma(fa, n1, cy);
    const float4 ob = __ldg(reinterpret_cast<const float4*>(d.key_obs_ff + 2LL * k));
    ff e0f = ff_add(u, ff_neg(ff{ob.x, ob.y})), e1f = ff_add(v, ff_neg(ff{ob.z, ob.w}));   // r = f(x) - y
    {
      const float r0 = e0f.hi + e0f.lo, r1 = e1f.hi + e1f.lo;
      acc_raw += double(fmaf(r0, r0, r1 * r1));
    }
    if (d.key_wl) {   // whitened residual L^T r
      const ff l00 = ff_ld(ff_split(__ldg(d.key_wl + 3LL * k)));
      const ff l10 = ff_ld(ff_split(__ldg(d.key_wl + 3LL * k + 1)));
      const ff l11 = ff_ld(ff_split(__ldg(d.key_wl + 3LL * k + 2)));
      const ff w0 = ff_fma(l00, e0f, ff_mul(l10, e1f));
      e1f = ff_mul(l11, e1f);
      e0f = w0;
    }
    const ff sqf = ff_fma(e0f, e0f, ff_mul(e1f, e1f));
    const float e0 = e0f.hi + e0f.lo, e1 = e1f.hi + e1f.lo;
    float sw = 1.0f;
    const float hd = float(d.huber_delta);
    if (d.loss == GBA_LOSS_HUBER && sqf.hi > hd * hd) {
      const float r = sqrtf(sqf.hi);
      acc = ff_add_f(acc, 2.0f * hd * r - hd * hd);
      sw = sqrtf(hd / r);
    } else {
      acc = ff_add(acc, sqf);
    }
    if (local) {
      rws[k - ch.begin] = make_float4(e0 * sw, e1 * sw, sw, 0.0f);
    } else {
      const float out[4] = {e0 * sw, e1 * sw, sw, 0.0f};
      store_vec<4>(rw + 4LL * k, out);
    }
  }
  // the candidate's Jacobian records, used if it is accepted: a second pass
  // over the chunk (each thread its own keys and the residuals it just
  // kept), so the cost loop keeps its register count
  if (records) linearize_chunk<float>(d, ch, par, local ? rws : nullptr);
  double sums[2] = {double(acc.hi) + double(acc.lo), acc_raw};
  const double tot = block_sums<2>(sums, red);
  if (threadIdx.x < 2) d.key_chunk_sum[2LL * blockIdx.x + threadIdx.x] = tot;
  if (which == 1 && d.fold_ctrl) {   // the accept decision in the last CTA of the problem
    __shared__ int last;
    const int p = ch.prob;
    if (last_arrival(d.fold_count + 2 * p + 1,
                     d.prob_key_chunk_off[p + 1] - d.prob_key_chunk_off[p], &last))
      ctrl_accept_body<true>(d, p, red);
  }
}

// Keys whose products the point kernels keep in shared memory at a time (a
// chunk of 128 points has about 700; longer ones go in parts).
constexpr int kPointKeys = 768;

// Per point: V_p = sum J_p^T J_p, g_p = sum J_p^T r from its keys' records:
// the products a key to a thread, then added point by point in key order (as
// the back-substitution does).  FP32: bound by DRAM (68%) and by the loads in
// flight, so 48 registers for ten blocks an SM (512 windows 477 -> 460 us; 40
// and twelve blocks spill: 495).
template <typename T>
__global__ void __launch_bounds__(kPointChunk, sizeof(T) == sizeof(float) ? 10 : 0) k_point_reduce(DevPlan d) {
  constexpr int kCap = kPointKeys / 2;
  __shared__ unsigned long long red[2 * kPointChunk / 32];
  __shared__ T prod[9][kCap];
  const Chunk ch = d.pt_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (!st.relin || !st.active) return;
  const int pt = ch.begin + threadIdx.x;
  T vmax = T(0), gmax = T(0);
  T V[6] = {0, 0, 0, 0, 0, 0}, g[3] = {0, 0, 0};
  {
    const T* __restrict__ JR = tptr<T>(d.JR[st.parity]);
    const int k0 = __ldg(d.pt_key_off + ch.begin), k1 = __ldg(d.pt_key_off + ch.end);
    const int kb = pt < ch.end ? __ldg(d.pt_key_off + pt) : k1, ke = pt < ch.end ? __ldg(d.pt_key_off + pt + 1) : k1;
    for (int base = k0; base < k1; base += kCap) {
      const int top = min(k1, base + kCap);
      for (int k = base + int(threadIdx.x); k < top; k += kPointChunk) {
        T jp[8], rr[2];
        load_vec<8>(JR + (long long)kJRStride * k, jp);
        load_vec<2>(JR + (long long)kJRStride * k + 18, rr);
        const int e = k - base;
        prod[0][e] = jp[0] * jp[0] + jp[3] * jp[3];
        prod[1][e] = jp[0] * jp[1] + jp[3] * jp[4];
        prod[2][e] = jp[0] * jp[2] + jp[3] * jp[5];
        prod[3][e] = jp[1] * jp[1] + jp[4] * jp[4];
        prod[4][e] = jp[1] * jp[2] + jp[4] * jp[5];
        prod[5][e] = jp[2] * jp[2] + jp[5] * jp[5];
        prod[6][e] = jp[0] * rr[0] + jp[3] * rr[1];
        prod[7][e] = jp[1] * rr[0] + jp[4] * rr[1];
        prod[8][e] = jp[2] * rr[0] + jp[5] * rr[1];
      }
      __syncthreads();
      const int e1 = min(ke, top) - base;
      for (int e = max(kb, base) - base; e < e1; ++e) {
#pragma unroll
        for (int c = 0; c < 6; ++c) V[c] += prod[c][e];
#pragma unroll
        for (int c = 0; c < 3; ++c) g[c] += prod[6 + c][e];
      }
      if (top < k1) __syncthreads();
    }
  }
  if (pt < ch.end) {
    if (d.pt_cons_off) {   // soft constraints: weight on the diagonal, w (x - y) in g
      const double* xp = d.x_pt[st.parity] + 3LL * pt;
      for (int c = d.pt_cons_off[pt]; c < d.pt_cons_off[pt + 1]; ++c) {
        const int row = d.cons_by_pt[c];
        const int b = d.cons[row].z;
        const double2 yw = d.cons_yw[row];
        V[b == 0 ? 0 : (b == 1 ? 3 : 5)] += T(yw.y);
        g[b] += T(yw.y * (xp[b] - yw.x));
      }
    }
    if (d.pt_prior_off) {   // point priors: V += L (its symmetric part), g += L (x - y)
      // (ba_gcp_constrained_normal_equation_builder.hpp:59-72)
      const double* xp = d.x_pt[st.parity] + 3LL * pt;
      for (int c = d.pt_prior_off[pt]; c < d.pt_prior_off[pt + 1]; ++c) {
        const int i = d.prior_by_pt[c];
        const double* L = d.prior_info + 9LL * i;
        const double v0 = xp[0] - d.prior_y[3LL * i], v1 = xp[1] - d.prior_y[3LL * i + 1],
                     v2 = xp[2] - d.prior_y[3LL * i + 2];
        V[0] += T(L[0]);
        V[1] += T(0.5 * (L[1] + L[3]));
        V[2] += T(0.5 * (L[2] + L[6]));
        V[3] += T(L[4]);
        V[4] += T(0.5 * (L[5] + L[7]));
        V[5] += T(L[8]);
        g[0] += T(L[0] * v0 + L[1] * v1 + L[2] * v2);
        g[1] += T(L[3] * v0 + L[4] * v1 + L[5] * v2);
        g[2] += T(L[6] * v0 + L[7] * v1 + L[8] * v2);
      }
    }
    T pv[12] = {V[0], V[1], V[2], V[3], V[4], V[5], g[0], g[1], g[2], T(0), T(0), T(0)};
    store_vec<12>(tptr_mut<T>(d.PV) + 12LL * pt, pv);
    vmax = fmax(fmax(V[0], V[3]), V[5]);
    gmax = fmax(fmax(fabs(g[0]), fabs(g[1])), fabs(g[2]));
  }
  LMState* sp = d.state + ch.prob;
  block_max2(vmax, gmax, red, &sp->maxdiag_bits, &sp->ginf_bits);
}

// image reduce: U_i = sum J_i^T J_i, g_i = sum J_i^T r.  Each image's keys
// are split into work items (one warp each) whose lanes add with
// compensation; k_image_finalize adds an image's items in FP64.
//
// FP32: Kahan, its order of operations part of the mixed path's results.
// FP64 (the pipe takes 64 cycles an instruction): the compensation enters the
// products' FMA chain, and a lane's keys are taken two to a compensated
// addition (3.5 instructions a key and entry instead of Kahan's 6), the carry
// register holding the first key's products; every key is folded in items
// of more than 256 keys (a caller's image_item) and in an image's only item.
// The tree's last addition keeps its rounding error, which k_image_finalize
// adds again.  Error against exact sums, root mean square relative to the sum
// of magnitudes (Kahan lanes over 512-key items added in order in
// parentheses): signed terms, 500 keys an image 6.8e-18 (7.1e-18), 5,000
// 2.2e-18 (2.9e-18), 20,000 1.1e-18 (2.1e-18); positive terms 5.0e-17
// (7.1e-17), 5.3e-17 (1.1e-16), 5.3e-17 (1.9e-16).  Plain FMA chains were as
// good for positive terms but up to 20% (default items) and 3.6 times
// (4,096-key items) worse for signed ones; the compensation takes 24 FP64
// windows from 19.1 to 19.6 ms a solve of 12 iterations.
// ---------------------------------------------------------------------------
enum AddMode { kAddChain, kAddFirst, kAddFold };   // FP64: carry on, start the sum, fold into it

template <AddMode kMode>
__device__ __forceinline__ void add_dot2(float& acc, float& cmp, float x0, float y0, float x1, float y1) {
  const float term = x0 * y0 + x1 * y1;
  const float y = term - cmp;
  const float t = acc + y;
  cmp = (t - acc) - y;
  acc = t;
}
// (cmp: what acc lacks, to be added)
template <AddMode kMode>
__device__ __forceinline__ void add_dot2(double& acc, double& cmp, double x0, double y0, double x1, double y1) {
  const double y = fma(x1, y1, fma(x0, y0, cmp));
  if constexpr (kMode == kAddFold) {
    const double t = acc + y;
    cmp = y - (t - acc);
    acc = t;
  } else if constexpr (kMode == kAddFirst) {   // (acc is 0: the same)
    acc = y;
    cmp = 0.0;
  } else {
    cmp = y;
  }
}
// a + b = s + e exactly
__device__ __forceinline__ double two_sum(double a, double b, double& e) {
  const double s = a + b, bb = s - a;
  e = (a - (s - bb)) + (b - bb);
  return s;
}

// One key's products into the 27 sums; v: its record from value 4 on.
template <AddMode kMode, typename T>
__device__ __forceinline__ void add_image_key(T* acc, T* cmp, const T* v) {
  const T* ji = v + 2;
  const T r0 = v[14], r1 = v[15];
  int e = 0;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
#pragma unroll
    for (int b = a; b < 6; ++b) {
      add_dot2<kMode>(acc[e], cmp[e], ji[a], ji[b], ji[6 + a], ji[6 + b]);
      ++e;
    }
  }
#pragma unroll
  for (int a = 0; a < 6; ++a) add_dot2<kMode>(acc[21 + a], cmp[21 + a], ji[a], r0, ji[6 + a], r1);
}

template <typename T>
__global__ void __launch_bounds__(256) k_image_reduce(DevPlan d) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= d.n_img_items) return;
  const int4 it = __ldg(d.img_items + wid);   // (image, q begin, q end, prob)
  const LMState& st = d.state[it.w];
  if (!st.relin || !st.active) return;
  const T* __restrict__ JR = tptr<T>(d.JR[st.parity]);
  T acc[27], cmp[27];
#pragma unroll
  for (int e = 0; e < 27; ++e) { acc[e] = T(0); cmp[e] = T(0); }
  // two loads deep: the key two rounds ahead and the record of the next round
  // are on their way while this one is added (the loads are scattered, and
  // a lane has nothing else to wait with: 11 of 14 cycles an instruction;
  // 512 windows 685 -> 517 us, random walk 274 -> 216)
  constexpr int kUse = kJRStride - 4;   // from value 4: J_i (6..17), r (18, 19)
  T next[kUse];
  int q = it.y + lane;
  int kn = q < it.z ? __ldg(d.img_keys + q) : 0;
  if (q < it.z) load_vec<kUse>(JR + (long long)kJRStride * kn + 4, next);
  kn = q + 32 < it.z ? __ldg(d.img_keys + q + 32) : kn;
  // (FP64) fold every key: long lanes, and an image's only item
  const bool whole = it.z - it.y > 256 || __ldg(d.img_item_off + it.x + 1) - __ldg(d.img_item_off + it.x) == 1;
  bool chain = false, first = true;   // the last key's products wait in cmp; no sum yet
  for (; q < it.z; q += 32) {
    T rec[kUse];
#pragma unroll
    for (int e = 0; e < kUse; ++e) rec[e] = next[e];
    if (q + 32 < it.z) load_vec<kUse>(JR + (long long)kJRStride * kn + 4, next);
    if (q + 64 < it.z) kn = __ldg(d.img_keys + q + 64);
    if constexpr (sizeof(T) == sizeof(float)) {
      add_image_key<kAddFold>(acc, cmp, rec);
    } else if (!chain && !whole) {
      add_image_key<kAddChain>(acc, cmp, rec);
      chain = true;
    } else {
      if (first)
        add_image_key<kAddFirst>(acc, cmp, rec);
      else
        add_image_key<kAddFold>(acc, cmp, rec);
      first = chain = false;
    }
  }
  int base, count;
  if constexpr (sizeof(T) == sizeof(float)) {
#pragma unroll
    for (int e = 0; e < 27; ++e) acc[e] -= cmp[e];
    warp_scatter_sums<27>(acc, lane, base, count);
    if (count > 0) d.img_item_partial[kImageItemStride<T> * wid + base] = double(acc[0]);
  } else {
    if (whole || it.z - it.y != 64) {   // (two keys a lane, chained: all of it is in acc)
#pragma unroll
      for (int e = 0; e < 27; ++e) acc[e] += cmp[e];
    }
    warp_scatter_sums<27, 16, 2>(acc, lane, base, count);
    // the last level: of the (up to) two values, one kept and one given
    const bool up = (lane & 1) != 0;
    const T keep = up ? acc[1] : acc[0], give = up ? acc[0] : acc[1];
    T lo;
    const T hi = two_sum(keep, __shfl_xor_sync(0xffffffffu, give, 1), lo);
    if (up ? count == 2 : count > 0) {
      double* out = d.img_item_partial + kImageItemStride<T> * wid + base + (up ? 1 : 0);
      out[0] = hi;
      out[28] = lo;
    }
  }
}

// An image's items added up.  Mixed: a warp an image, the items in order.  FP64
// (finer items, image_item_size): four interleaved compensated sums, a warp
// each: five dependent additions an item at 64 cycles each, so with all four
// in one warp and eight images to a CTA a window alone (40 items an image) took
// 17 us longer a launch, 512 windows one after the other 283 solves/s instead of
// 299.
constexpr int kFinalizeThreads = 128;   // FP64: a CTA an image

template <typename T>
__global__ void __launch_bounds__(256) k_image_finalize(DevPlan d) {
  constexpr bool kWhole = sizeof(T) == sizeof(double);
  constexpr long long kStride = kImageItemStride<T>;
  __shared__ double sums[kWhole ? 4 : 1][2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int img = kWhole ? int(blockIdx.x) : int(blockIdx.x) * 8 + warp;
  if (img >= d.I) return;
  const int prob = d.img_prob[img];
  const LMState& st = d.state[prob];
  if (!st.relin || !st.active) return;
  const int ib = d.img_item_off[img], ie = d.img_item_off[img + 1];
  const double* part = d.img_item_partial + min(lane, 26);
  double v = 0.0;
  if constexpr (!kWhole) {
    if (lane < 27)
      for (int t = ib; t < ie; ++t) v += part[kStride * t];
  } else {
    double s = 0.0, c = 0.0;
    for (int t0 = ib + warp; t0 < ie; t0 += 16) {
      double hi[4], lo[4];   // (the loads of four items together)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = min(t0 + 4 * u, ie - 1);
        hi[u] = part[kStride * t];
        lo[u] = part[kStride * t + 28];
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (u == 0 && t0 == ib + warp) {
          s = hi[0];
          c = lo[0];
        } else if (t0 + 4 * u < ie) {
          const double y = hi[u] + c, n = s + y;
          c = (y - (n - s)) + lo[u];
          s = n;
        }
      }
    }
    sums[warp][0][lane] = s;
    sums[warp][1][lane] = c;
    __syncthreads();
    if (warp > 0) return;
    double e0, e1, e2;
    const double a = two_sum(sums[0][0][lane], sums[1][0][lane], e0),
                 b = two_sum(sums[2][0][lane], sums[3][0][lane], e1);
    v = two_sum(a, b, e2);
    v += ((sums[0][1][lane] + sums[1][1][lane]) + (sums[2][1][lane] + sums[3][1][lane])) + ((e0 + e1) + e2);
  }
  // lane e holds entry e of (upper U in row order, then g)
  double* U = d.U + 36LL * img;
  double dmax = 0.0, gmax = 0.0;
  if (d.img_cons_off && lane < 27) {   // soft constraints on this image's parameters
    int a = -1, b = -1;
    if (lane < 21) {
      int e = lane;
      a = 0;
      while (e >= 6 - a) { e -= 6 - a; ++a; }
      b = a + e;
    }
    const double* xi = d.x_img[st.parity] + 6LL * img;
    for (int c = d.img_cons_off[img]; c < d.img_cons_off[img + 1]; ++c) {
      const int row = d.cons_by_img[c];
      const int prm = d.cons[row].z;
      const double2 yw = d.cons_yw[row];
      if (lane < 21 && a == b && a == prm) v += yw.y;
      if (lane >= 21 && lane - 21 == prm) v += yw.y * (xi[prm] - yw.x);
    }
  }
  if (lane < 21) {
    int a = 0, e = lane;
    while (e >= 6 - a) { e -= 6 - a; ++a; }
    const int b = a + e;
    U[6 * a + b] = v;
    U[6 * b + a] = v;
    if (a == b) dmax = v;
  } else if (lane < 27) {
    d.gi[6LL * img + (lane - 21)] = v;
    gmax = fabs(v);
  }
  dmax = warp_max(dmax);
  gmax = warp_max(gmax);
  if (lane == 0) {
    LMState* sp = d.state + prob;
    atomicMax(&sp->maxdiag_bits, dbits(dmax));
    atomicMax(&sp->ginf_bits, dbits(gmax));
  }
}

// ---------------------------------------------------------------------------
// Free cameras: per image work item (the items of k_image_reduce) the sums
// E = J_i^T J_c (6 x 10), the upper triangle of J_c^T J_c (55) and J_c^T r
// (10) over its keys (camera_shared_normal_equation_builder.hpp:111-462 for
// the camera blocks).  A CTA stages 32 keys' rows [J_i | J_c | r] in shared
// memory; thread e owns sum e (each batch in T, batches added in FP64, keys
// in order).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_image_cam_reduce(DevPlan d) {
  __shared__ T M[64][17];
  const int4 it = d.img_items[blockIdx.x];   // (image, q begin, q end, prob)
  const LMState& st = d.state[it.w];
  if (!st.relin || !st.active) return;
  if (d.cam_info[d.img_cam[it.x]].x == 0) return;
  const T* __restrict__ JR = tptr<T>(d.JR[st.parity]);
  const T* __restrict__ JC = tptr<T>(d.JC[st.parity]);
  const int e = threadIdx.x;
  int ca = 0, cb = 0;
  if (e < 60) {
    ca = e / 10;
    cb = 6 + e % 10;
  } else if (e < 115) {
    int t = e - 60, m = 0;
    while (t >= 10 - m) {
      t -= 10 - m;
      ++m;
    }
    ca = 6 + m;
    cb = 6 + m + t;
  } else if (e < 125) {
    ca = 6 + (e - 115);
    cb = 16;
  }
  double acc = 0.0;
  for (int q0 = it.y; q0 < it.z; q0 += 32) {
    const int nq = min(32, it.z - q0);
    if (threadIdx.x < 64) {   // thread r stages row r: key r/2, Jacobian row r%2
      const int row = threadIdx.x, kq = row >> 1, rr = row & 1;
      T v[17];
#pragma unroll
      for (int c = 0; c < 17; ++c) v[c] = T(0);
      if (kq < nq) {
        const long long k = __ldg(d.img_keys + q0 + kq);
        const T* jr = JR + kJRStride * k;
        const T* jc = JC + 20 * k + 10 * rr;
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = jr[6 + 6 * rr + c];
#pragma unroll
        for (int c = 0; c < 10; ++c) v[6 + c] = jc[c];
        v[16] = jr[18 + rr];
      }
#pragma unroll
      for (int c = 0; c < 17; ++c) M[row][c] = v[c];
    }
    __syncthreads();
    if (e < 125) {   // 32 keys in T, then into the FP64 total in key order
      T bs = T(0);
      for (int row = 0; row < 2 * nq; ++row) bs = fma(M[row][ca], M[row][cb], bs);
      acc += double(bs);
    }
    __syncthreads();
  }
  d.img_item_cam[(long long)kImgCamVals * blockIdx.x + e] = e < 125 ? acc : 0.0;
}

// Per image with a free camera: the FP64 sums of its work items' partials
// (items in order); E_i also goes to its own array for the assembly.
__global__ void __launch_bounds__(kImgCamVals) k_image_cam_finalize(DevPlan d) {
  const int img = blockIdx.x;
  const int4 ci = d.cam_info[d.img_cam[img]];
  if (ci.x == 0) return;
  const LMState& st = d.state[ci.z];
  if (!st.relin || !st.active) return;
  const int e = threadIdx.x;
  double v = 0.0;
  for (int t = d.img_item_off[img]; t < d.img_item_off[img + 1]; ++t)
    v += d.img_item_cam[(long long)kImgCamVals * t + e];
  d.img_cam_sum[(long long)kImgCamVals * img + e] = v;
  if (e < 60) d.Ei[60LL * img + e] = v;
}

// Per free camera: U_c and g_c summed over its images in FP64 (kCamGroups
// groups of kImgCamVals threads take every kCamGroups-th image in order, the
// group sums are added in group order), compacted to the computed
// parameters, with the camera's soft constraints
// (camera_shared_normal_equation_builder.hpp:309-349,418-459).
constexpr int kCamGroups = 8;
__global__ void __launch_bounds__(kImgCamVals * kCamGroups) k_cam_finalize(DevPlan d) {
  __shared__ double part[kCamGroups][kImgCamVals];
  __shared__ double sh[kImgCamVals];
  const int c = blockIdx.x;
  const int4 ci = d.cam_info[c];
  if (ci.x == 0) return;
  const LMState& st = d.state[ci.z];
  if (!st.relin || !st.active) return;
  const int e = threadIdx.x % kImgCamVals, grp = threadIdx.x / kImgCamVals;
  double tot = 0.0;
  for (int u = d.cam_img_off[c] + grp; u < d.cam_img_off[c + 1]; u += kCamGroups)
    tot += d.img_cam_sum[(long long)kImgCamVals * d.cam_imgs[u] + e];
  part[grp][e] = tot;
  __syncthreads();
  if (threadIdx.x < kImgCamVals) {
    double v = 0.0;
#pragma unroll
    for (int g = 0; g < kCamGroups; ++g) v += part[g][e];
    sh[e] = v;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  const int cps = ci.x;
  const unsigned mask = unsigned(ci.y);
  double* U = d.Uc + 100LL * c;
  double* g = d.gc + 10LL * c;
  for (int m = 0; m < cps; ++m) {
    const int fm = cam_full_col(mask, m);
    for (int n = 0; n < cps; ++n) {
      const int fn = cam_full_col(mask, n);
      U[10 * m + n] = sh[60 + upper10(min(fm, fn), max(fm, fn))];
    }
    g[m] = sh[115 + fm];
  }
  if (d.n_cons > 0) {
    const double* x = d.x_cam[st.parity] + 10LL * c;
    for (int r = d.prob_cons_off[ci.z]; r < d.prob_cons_off[ci.z + 1]; ++r) {
      const int4 cr = d.cons[r];
      if (cr.x != 2 || cr.y != c) continue;
      const double2 yw = d.cons_yw[r];
      U[11 * cr.z] += yw.y;
      g[cr.z] += yw.y * (x[cr.z] - yw.x);
    }
  }
  double dmax = 0.0, gmax = 0.0;
  for (int m = 0; m < cps; ++m) {
    dmax = fmax(dmax, U[11 * m]);
    gmax = fmax(gmax, fabs(g[m]));
  }
  LMState* sp = d.state + ci.z;
  atomicMax(&sp->maxdiag_bits, dbits(dmax));
  atomicMax(&sp->ginf_bits, dbits(gmax));
}

// ---------------------------------------------------------------------------
// point factor: C C^T = V_p + mu I, C^-1 and h_p = C^-1 g_p per point
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kPointChunk) k_point_factor(DevPlan d) {
  const Chunk ch = d.pt_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (!st.active) return;
  const int pt = ch.begin + threadIdx.x;
  if (pt >= ch.end) return;
  const T mu = T(st.mu);
  T pv[12];
  load_vec<12>(tptr<T>(d.PV) + 12LL * pt, pv);
  const T a00 = pv[0] + mu, a01 = pv[1], a02 = pv[2], a11 = pv[3] + mu, a12 = pv[4], a22 = pv[5] + mu;
  bool ok = a00 > T(0);
  const T c00 = sqrt(a00);
  const T i00 = T(1) / c00;
  const T c10 = a01 * i00, c20 = a02 * i00;
  const T s11 = a11 - c10 * c10;
  ok = ok && s11 > T(0);
  const T c11 = sqrt(s11);
  const T i11 = T(1) / c11;
  const T c21 = (a12 - c20 * c10) * i11;
  const T s22 = a22 - c20 * c20 - c21 * c21;
  ok = ok && s22 > T(0);
  const T c22 = sqrt(s22);
  const T i22 = T(1) / c22;
  if (!ok) {
    atomicExch(d.factor_flag + ch.prob, 1);
    return;
  }
  // C^-1 (lower): rows [i00 0 0; m10 i11 0; m20 m21 i22]
  const T m10 = -c10 * i00 * i11;
  const T m21 = -c21 * i11 * i22;
  const T m20 = -(c20 * i00 + c21 * m10) * i22;
  const T g0 = pv[6], g1 = pv[7], g2 = pv[8];
  T ps[12] = {i00, m10, i11, m20, m21, i22,
              i00 * g0, m10 * g0 + i11 * g1, m20 * g0 + m21 * g1 + i22 * g2, T(0), T(0), T(0)};
  store_vec<12>(tptr_mut<T>(d.PS) + 12LL * pt, ps);
}

// Z_a = C_p^-1 J_p^T J_i per key, one slot per thread: slot s holds key s
// (records) or key img_keys[s], the keys image by image (planes), so the
// writes are coalesced either way.  DevPlan::key_z_split CTAs share each
// key chunk (a problem's slots are its keys' range), so the grid fills the
// GPU in even waves.
template <typename T>
__global__ void __launch_bounds__(256) k_key_z(DevPlan d) {
  const int split = d.key_z_split;
  const Chunk ch = d.key_chunks[blockIdx.x / split];
  const LMState& st = d.state[ch.prob];
  if (!st.active) return;
  const T* __restrict__ JR = tptr<T>(d.JR[st.parity]);
  const T* __restrict__ PS = tptr<T>(d.PS);
  T* __restrict__ Z = tptr_mut<T>(d.Z);
  const int sub = blockIdx.x % split;
  for (int sl = ch.begin + sub * 256 + threadIdx.x; sl < ch.end; sl += split * 256) {
    const int k = d.z_planes ? __ldg(d.img_keys + sl) : sl;
    T rec[kJRStride], ps[8];
    load_vec<kJRStride>(JR + (long long)kJRStride * k, rec);
    load_vec<8>(PS + 12LL * __ldg(d.key_pt + k), ps);
    const T i00 = ps[0], m10 = ps[1], i11 = ps[2], m20 = ps[3], m21 = ps[4], i22 = ps[5];
    const T* jp = rec;
    const T* ji = rec + 6;
    T z[kZStride];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const T w0 = jp[0] * ji[c] + jp[3] * ji[6 + c];
      const T w1 = jp[1] * ji[c] + jp[4] * ji[6 + c];
      const T w2 = jp[2] * ji[c] + jp[5] * ji[6 + c];
      z[c] = i00 * w0;
      z[6 + c] = m10 * w0 + i11 * w1;
      z[12 + c] = m20 * w0 + m21 * w1 + i22 * w2;
    }
    z[18] = T(0);
    z[19] = T(0);
    store_z(d, Z, sl, z);
  }
}

// Free cameras: per camera record r of a point (camera c, part h) the Z
// record C_p^-1 W with W = sum over the point's keys seen through camera c
// of J_p^T J_c[:, 6h .. 6h+5] (computed parameters; zero past them).  The
// records of one camera are consecutive; one pass over the point's keys
// builds all of them (W for up to 12 computed columns).
template <typename T>
__global__ void __launch_bounds__(kPointChunk) k_camrec_z(DevPlan d) {
  const Chunk ch = d.pt_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (!st.active) return;
  const int pt = ch.begin + threadIdx.x;
  if (pt >= ch.end) return;
  const int rb = d.pt_rec_off[pt], re = d.pt_rec_off[pt + 1];
  if (rb == re) return;
  const T* __restrict__ JR = tptr<T>(d.JR[st.parity]);
  const T* __restrict__ JC = tptr<T>(d.JC[st.parity]);
  T ps[8];
  load_vec<8>(tptr<T>(d.PS) + 12LL * pt, ps);
  const T i00 = ps[0], m10 = ps[1], i11 = ps[2], m20 = ps[3], m21 = ps[4], i22 = ps[5];
  const int kb = d.pt_key_off[pt], ke = d.pt_key_off[pt + 1];
  for (int r = rb; r < re;) {
    const int cam = d.rec_info[r - d.K].x;
    const int4 ci = d.cam_info[cam];
    const int nparts = (ci.x + 5) / 6;
    // W (3 x 12): the full-column index of each computed parameter
    T w[36];
#pragma unroll
    for (int e = 0; e < 36; ++e) w[e] = T(0);
    for (int k = kb; k < ke; ++k) {
      if (__ldg(d.img_cam + __ldg(d.key_img + k)) != cam) continue;
      T jp[8], jc[20];
      load_vec<8>(JR + (long long)kJRStride * k, jp);
      load_vec<20>(JC + 20LL * k, jc);
#pragma unroll
      for (int m = 0; m < 12; ++m) {
        if (m >= ci.x) break;
        const int f = cam_full_col(unsigned(ci.y), m);
        T j0 = T(0), j1 = T(0);
#pragma unroll
        for (int q = 0; q < 10; ++q)
          if (q == f) {
            j0 = jc[q];
            j1 = jc[10 + q];
          }
#pragma unroll
        for (int i = 0; i < 3; ++i) w[12 * i + m] += jp[i] * j0 + jp[3 + i] * j1;
      }
    }
    for (int h = 0; h < nparts; ++h, ++r) {
      T z[kZStride];
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        T w0 = T(0), w1 = T(0), w2 = T(0);
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          if (hh == h) {
            w0 = w[6 * hh + a];
            w1 = w[12 + 6 * hh + a];
            w2 = w[24 + 6 * hh + a];
          }
        z[a] = i00 * w0;
        z[6 + a] = m10 * w0 + i11 * w1;
        z[12 + a] = m20 * w0 + m21 * w1 + i22 * w2;
      }
      z[18] = T(0);
      z[19] = T(0);
      store_z(d, tptr_mut<T>(d.Z), r, z);
    }
  }
}

// Plan build, Z planes: the slot of every key (the inverse of img_keys) ...
__global__ void __launch_bounds__(256) k_key_slots(const int* __restrict__ img_keys, int K, int* __restrict__ key_slot) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < K) key_slot[img_keys[s]] = s;
}

// ... and the key pairs of the assembly's work items as slots (a camera
// record's index, >= K, is its slot; a diagonal block's second entry is
// the point and stays).
__global__ void __launch_bounds__(128) k_pairs_to_slots(const int4* __restrict__ items, int n_items,
                                                        const int2* __restrict__ blk_ij,
                                                        const int* __restrict__ key_slot, int K,
                                                        int2* __restrict__ pairs) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= n_items) return;
  const int4 it = items[wid];
  const int2 ij = blk_ij[it.x];
  const bool diag = ij.x == ij.y;
  for (int q = it.y + lane; q < it.z; q += 32) {
    int2 pr = pairs[q];
    pr.x = pr.x < K ? key_slot[pr.x] : pr.x;
    if (!diag) pr.y = pr.y < K ? key_slot[pr.y] : pr.y;
    pairs[q] = pr;
  }
}

// ---------------------------------------------------------------------------
// Schur assembly, one warp per work item (<= kPairItem pairs of one block)
// ---------------------------------------------------------------------------
// acc += x0 y0 + x1 y1 + x2 y2.  In FP64 one chain of three FMAs (three
// instructions at 64 cycles each on this part's FP64 pipe instead of a
// product, two FMAs and an addition: 24 windows 19.7 ms a solve against 22.2,
// the grid 48 against 54, their results as far from 64-bit references either
// way; a sum of 190 signed triples alone is off by 1.2e-17 of the sum of
// magnitudes, root mean square, against 1.05e-17); in FP32 the products first,
// the order the mixed path's results are defined by.
__device__ __forceinline__ void add_dot3(float& acc, float x0, float y0, float x1, float y1, float x2, float y2) {
  acc += x0 * y0 + x1 * y1 + x2 * y2;
}
__device__ __forceinline__ void add_dot3(double& acc, double x0, double y0, double x1, double y1, double x2,
                                         double y2) {
  acc = fma(x2, y2, fma(x1, y1, fma(x0, y0, acc)));
}

// The FP32 items are bound by the 16-byte gathers of their records through
// L1, the FP64 items by the FP64 pipe.  A diagonal block is symmetric: its 21
// upper sums are formed and mirrored (the products commute, so the same
// bits).  The 42 sums of an item are reduced by warp_scatter_sums (43
// additions instead of 210: at 190 pairs an item the reduction was a fifth
// of the FP64 instructions).  Measured over whole solves, all of it: FP64 grid
// (200 cameras, 3.9 M pairs, 20,791 items; 19 iterations) 80.9 -> 71.4 ms, 24
// FP64 windows 35.6 -> 30.6 ms; mixed grid 12.21 -> 11.99 ms.
template <typename T>
__global__ void __launch_bounds__(128) k_assemble_items(DevPlan d, int n_items) {
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= n_items) return;
  const int4 it = __ldg(d.items + wid);
  // the problem's state, the block and the first pair are independent
  // loads: all three are issued before the first of them is used
  const int active = d.state[it.w].active;
  const int2 ij = __ldg(d.blk_ij + it.x);
  int q = it.y + lane;
  int2 pr = q < it.z ? __ldg(d.pairs + q) : make_int2(0, 0);
  if (!active) return;
  const bool diag = ij.x == ij.y;
  const T* __restrict__ Z = tptr<T>(d.Z);
  const T* __restrict__ PS = tptr<T>(d.PS);
  T sum[42];   // the block's 36 entries, then the rhs' 6
#pragma unroll
  for (int e = 0; e < 42; ++e) sum[e] = T(0);
  // the next pair's key indices are fetched one iteration ahead, so each
  // iteration waits on a single round trip (the Z records)
  if (diag) {
    for (; q < it.z; q += 32) {
      const int qn = q + 32;
      const int2 prn = qn < it.z ? __ldg(d.pairs + qn) : pr;
      T z[kZStride], ps[8];
      load_z(d, Z, pr.x, z);
      load_vec<8>(PS + 12LL * pr.y + 4, ps);   // a diagonal block's pair carries the point; h = ps[2..4]
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        sum[36 + r] += z[r] * ps[2] + z[6 + r] * ps[3] + z[12 + r] * ps[4];
#pragma unroll
        for (int c = r; c < 6; ++c) add_dot3(sum[6 * r + c], z[r], z[c], z[6 + r], z[6 + c], z[12 + r], z[12 + c]);
      }
      pr = prn;
    }
#pragma unroll
    for (int r = 1; r < 6; ++r)
#pragma unroll
      for (int c = 0; c < r; ++c) sum[6 * r + c] = sum[6 * c + r];
  } else {
    for (; q < it.z; q += 32) {
      const int qn = q + 32;
      const int2 prn = qn < it.z ? __ldg(d.pairs + qn) : pr;
      T za[kZStride], zb[kZStride];
      load_z(d, Z, pr.x, za);
      load_z(d, Z, pr.y, zb);
#pragma unroll
      for (int r = 0; r < 6; ++r) {
#pragma unroll
        for (int c = 0; c < 6; ++c)
          add_dot3(sum[6 * r + c], za[r], zb[c], za[6 + r], zb[6 + c], za[12 + r], zb[12 + c]);
      }
      pr = prn;
    }
  }
  // reduced in the working precision, stored in FP64 by the lanes that end
  // with the sums
  int base, count;
  warp_scatter_sums<42>(sum, lane, base, count);
  double* out = d.item_partial + (long long)kItemStride * wid + base;
#pragma unroll
  for (int e = 0; e < warp_scatter_max(42); ++e)
    if (e < count) out[e] = double(sum[e]);
}

// Sum of one entry over work items [ib, ie) (stride kItemStride): in order
// for short lists; else items t = ib + 4u + r go to partial r and the
// partials are added in order (four loads in flight).
__device__ __forceinline__ double sum_items4(const double* base, int ib, int ie) {
  if (ie - ib < 8) {   // the common short lists: in order
    double v = 0.0;
    for (int t = ib; t < ie; ++t) v += base[(long long)kItemStride * t];
    return v;
  }
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  int t = ib;
  for (; t + 4 <= ie; t += 4) {
    s0 += base[(long long)kItemStride * t];
    s1 += base[(long long)kItemStride * (t + 1)];
    s2 += base[(long long)kItemStride * (t + 2)];
    s3 += base[(long long)kItemStride * (t + 3)];
  }
  if (t < ie) s0 += base[(long long)kItemStride * t];
  if (t + 1 < ie) s1 += base[(long long)kItemStride * (t + 1)];
  if (t + 2 < ie) s2 += base[(long long)kItemStride * (t + 2)];
  return (s0 + s1) + (s2 + s3);
}

// The entry (row 6i + a, column 6j + bcol), i >= j, of a problem's reduced
// system before the Schur terms and the damping (i, j local reduced-system
// images: the images, then each free camera's parts): U_i on an image's
// diagonal block, E_i between an image and the parts of its camera, U_c
// between parts of one camera; zero past a camera's parameters.
__device__ __forceinline__ double reduced_base(const DevPlan& d, const ProbInfo& pi, int i, int a, int j,
                                               int bcol) {
  const int ni = pi.num_images;
  if (i < ni) return i == j ? d.U[36LL * (pi.image_begin + i) + 6 * a + bcol] : 0.0;
  // camera part: global camera ci, parameter m of the row
  const int ci = pi.cam_begin + (i - ni) / pi.nc;
  const int4 cinf = d.cam_info[ci];
  const int m = 6 * ((i - ni) % pi.nc) + a;
  if (m >= cinf.x) return 0.0;
  if (j >= ni) {
    const int cj = pi.cam_begin + (j - ni) / pi.nc;
    const int mj = 6 * ((j - ni) % pi.nc) + bcol;
    return (cj == ci && mj < cinf.x) ? d.Uc[100LL * ci + 10 * m + mj] : 0.0;
  }
  const int gj = pi.image_begin + j;
  return d.img_cam[gj] == ci ? d.Ei[60LL * gj + 10 * bcol + cam_full_col(unsigned(cinf.y), m)] : 0.0;
}

// The gradient entry of row 6i + a of the reduced system (g_i or g_c).
__device__ __forceinline__ double reduced_grad(const DevPlan& d, const ProbInfo& pi, int i, int a) {
  const int ni = pi.num_images;
  if (i < ni) return d.gi[6LL * (pi.image_begin + i) + a];
  const int ci = pi.cam_begin + (i - ni) / pi.nc;
  const int m = 6 * ((i - ni) % pi.nc) + a;
  return m < d.cam_info[ci].x ? d.gc[10LL * ci + m] : 0.0;
}

// Dense reduced system (lower triangle) and rhs in precision T; the block
// sums over work items are taken in FP64.  Rows and columns run over the
// problem's reduced-system images: its images, then with free cameras nc
// 6-wide parts of each camera (camera_shared_normal_equation_solver.hpp:270-392,
// 422-443: U_c, the image-camera blocks E and g_c enter as the images' U and
// g do; columns past the camera's parameters hold mu alone).
template <typename T>
__global__ void __launch_bounds__(256) k_assemble_S(DevPlan d) {
  const int p = blockIdx.y;
  const ProbInfo pi = d.prob[p];
  const LMState& st = d.state[p];
  if (!st.active) return;
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int n = pi.n;
  if (idx >= (long long)n * n) return;
  const int row = int(idx / n), col = int(idx % n);
  if (col > row) return;
  const int i = row / 6, a = row % 6, j = col / 6, bcol = col % 6;
  const int Ie = pi.num_ext, ni = pi.num_images;
  const int blk = __ldg(d.blk_map + d.blk_map_off[p] + (long long)j * Ie + i);
  double v = 0.0, rv = 0.0;
  if (blk >= 0) {   // four interleaved partial sums (loads in flight together), then in order
    const int ib = __ldg(d.blk_item_off + blk), ie = __ldg(d.blk_item_off + blk + 1);
    v = sum_items4(d.item_partial + 6 * bcol + a, ib, ie);
  }
  (void)ni;
  const double base = reduced_base(d, pi, i, a, j, bcol);
  const double g = col == 0 ? reduced_grad(d, pi, i, a) : 0.0;
  double s = base - v;
  if (row == col) s += st.mu;
  tptr_mut<T>(d.S)[pi.s_off + (long long)row * n + col] = T(s);
  if (col == 0) {
    // rhs b_i[a] = g_i[a] - sum over the diagonal block's items
    const int dblk = __ldg(d.blk_map + d.blk_map_off[p] + (long long)i * Ie + i);
    rv = 0.0;
    if (dblk >= 0) {
      const int ib = __ldg(d.blk_item_off + dblk), ie = __ldg(d.blk_item_off + dblk + 1);
      rv = sum_items4(d.item_partial + 36 + a, ib, ie);
    }
    tptr_mut<T>(d.b)[6LL * (pi.ext_begin + i) + a] = T(g - rv);
  }
}

// The same dense system, block by block (plans without free cameras): S is
// zeroed first (the entries of image pairs without a common point are 0)
// unless every image pair has a block (DevPlan::s_complete: nothing but the
// blocks is read of it; one graph node of about 3 us less), then one thread per entry of every block writes base - sum over the
// block's items (+ mu on the diagonal) exactly as k_assemble_S does, the 36
// threads of a block reading its items' partials together; the threads of
// row 0 of each diagonal block write the rhs.
template <typename T>
__global__ void __launch_bounds__(256) k_assemble_S_blocks(DevPlan d) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= 36LL * d.n_blocks) return;
  const int blk = int(e / 36), el = int(e % 36);
  const int p = __ldg(d.blk_prob + blk);
  const LMState& st = d.state[p];
  if (!st.active) return;
  const ProbInfo pi = d.prob[p];
  const int2 xy = __ldg(d.blk_ij + blk);   // column image x <= row image y
  const int a = el % 6, bcol = el / 6;     // partial entry 6 * bcol + a = el
  const int row = 6 * xy.y + a, col = 6 * xy.x + bcol;
  const int2 items = make_int2(__ldg(d.blk_item_off + blk), __ldg(d.blk_item_off + blk + 1));
  if (col <= row) {
    const double v = sum_items4(d.item_partial + el, items.x, items.y);
    const double base = reduced_base(d, pi, xy.y, a, xy.x, bcol);
    double s = base - v;
    if (row == col) s += st.mu;
    tptr_mut<T>(d.S)[pi.s_off + (long long)row * pi.n + col] = T(s);
  }
  if (xy.x == xy.y && bcol == 0) {   // rhs b_y[a] = g_y[a] - sum over the diagonal block's items
    const double rv = sum_items4(d.item_partial + 36 + a, items.x, items.y);
    const double g = reduced_grad(d, pi, xy.y, a);
    tptr_mut<T>(d.b)[6LL * (pi.ext_begin + xy.y) + a] = T(g - rv);
  }
}

// ---------------------------------------------------------------------------
// Tiled Cholesky of the reduced system S (lower, precision T), one launch per
// column step.  Launch k (k = -1 .. nt-2) subtracts column k's rank-32
// contribution from every trailing tile and factors column c = k+1: every
// CTA of column c recomputes the diagonal tile's factor and inverse itself
// (tile_potrf_inverse: three of its warps in FP32, four in FP64), so no separate
// panel launch is needed; the CTA owning tile (c, c) publishes L_cc^-1 and the
// forward-solve value y_c = L_cc^-1 b_c.  S keeps its diagonal tiles (the
// factor lives in Linv), the off-diagonal tiles are overwritten by L.
// The backward solve L^T delta = y then takes one launch per tile row.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int tile_rows(int n, int t) { return min(kTile, n - kTile * t); }

// Calls f(std::integral_constant<int, i>) for i = B, B + S, ... < E.
template <int B, int E, int S, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    static_for<B + S, E, S>(f);
  }
}

// Shared-memory tiles: rows padded to a 16-byte multiple (36 floats, 34
// doubles) so that 16-byte vector loads along a row are aligned and the
// rows touched together fall in different banks.
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
  using V = float4;
  static constexpr int N = 4;
  __device__ __forceinline__ static void unpack(const V& v, float* o) {
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
  __device__ __forceinline__ static V pack(const float* o) { return make_float4(o[0], o[1], o[2], o[3]); }
};
template <>
struct Vec16<double> {
  using V = double2;
  static constexpr int N = 2;
  __device__ __forceinline__ static void unpack(const V& v, double* o) {
    o[0] = v.x;
    o[1] = v.y;
  }
  __device__ __forceinline__ static V pack(const double* o) { return make_double2(o[0], o[1]); }
};

template <typename T>
using Tile = T[kTile][kTile + Vec16<T>::N];

// Tile loads for 256-thread CTAs: each thread fetches its 4 elements of a
// tile into registers first (all loads in flight together), then stores
// them to shared memory.  Rectangular tiles read 0 past the matrix; a
// diagonal tile keeps its stored lower triangle, reads 0 above it and has
// identity rows past the matrix.
constexpr int kCholThreads = 256;
constexpr int kPerThread = kTile * kTile / kCholThreads;

template <typename T>
struct TileFetch {
  T v[kPerThread];
  __device__ __forceinline__ void rect(const T* S, int n, int ti, int tj) {
    const int mi = tile_rows(n, ti), mj = tile_rows(n, tj);
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      const int e = threadIdx.x + u * kCholThreads, r = e / kTile, c = e % kTile;
      v[u] = (r < mi && c < mj) ? S[(long long)(kTile * ti + r) * n + kTile * tj + c] : T(0);
    }
  }
  __device__ __forceinline__ void diag(const T* S, int n, int ti) {
    const int m = tile_rows(n, ti);
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      const int e = threadIdx.x + u * kCholThreads, r = e / kTile, c = e % kTile;
      T x = T(0);
      if (r < m) {
        if (c <= r) x = S[(long long)(kTile * ti + r) * n + kTile * ti + c];
      } else if (r == c) {
        x = T(1);
      }
      v[u] = x;
    }
  }
  __device__ __forceinline__ void store(Tile<T>& t) const {
#pragma unroll
    for (int u = 0; u < kPerThread; ++u) {
      const int e = threadIdx.x + u * kCholThreads;
      t[e / kTile][e % kTile] = v[u];
    }
  }
};

// s[u] = sum_q X[r][q] Y[c][q] (q ascending) for the 128 threads tid < 128:
// rows r = tid / 8 and r + 16, columns c = tid % 8 + 8u (u = 0..3); s[0..3]
// is row r, s[4..7] row r + 16.  Rows are read with 16-byte vector loads; the
// rows a warp reads at once lie in distinct banks.  Two rows per thread halve
// the shared-memory wavefronts per FMA against one row per thread.
template <typename T>
__device__ __forceinline__ void tile_xyt_t(const Tile<T>& X, const Tile<T>& Y, T s[8], int t) {
  using V = Vec16<T>;
  constexpr int N = V::N;
  const int r = t >> 3, c0 = t & 7;
#pragma unroll
  for (int u = 0; u < 8; ++u) s[u] = T(0);
#pragma unroll
  for (int q = 0; q < kTile; q += N) {
    T x0[N], x1[N];
    V::unpack(*reinterpret_cast<const typename V::V*>(&X[r][q]), x0);
    V::unpack(*reinterpret_cast<const typename V::V*>(&X[r + 16][q]), x1);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      T y[N];
      V::unpack(*reinterpret_cast<const typename V::V*>(&Y[c0 + 8 * u][q]), y);
#pragma unroll
      for (int e = 0; e < N; ++e) {
        s[u] = fma(x0[e], y[e], s[u]);
        s[4 + u] = fma(x1[e], y[e], s[4 + u]);
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void tile_xyt(const Tile<T>& X, const Tile<T>& Y, T s[8]) {
  tile_xyt_t<T>(X, Y, s, threadIdx.x);
}

// A -= X Y^T (32x32x32) by the 128 threads t = 0..127 of a thread group, 8
// outputs each (the same outputs and sums for every group).
template <typename T>
__device__ __forceinline__ void tile_sub_xyt_t(Tile<T>& A, const Tile<T>& X, const Tile<T>& Y, int t) {
  T s[8];
  tile_xyt_t<T>(X, Y, s, t);
  const int r = t >> 3, c0 = t & 7;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    A[r][c0 + 8 * u] -= s[u];
    A[r + 16][c0 + 8 * u] -= s[4 + u];
  }
}

// A -= X Y^T (32x32x32) by threads 0..127, 8 outputs each.
template <typename T>
__device__ __forceinline__ void tile_sub_xyt(Tile<T>& A, const Tile<T>& X, const Tile<T>& Y) {
  if (threadIdx.x < 128) tile_sub_xyt_t<T>(A, X, Y, threadIdx.x);
}

__device__ __forceinline__ void load16(const float* p, float* o) {
  Vec16<float>::unpack(*reinterpret_cast<const float4*>(p), o);
}
__device__ __forceinline__ void load16(const double* p, double* o) {
  Vec16<double>::unpack(*reinterpret_cast<const double2*>(p), o);
}

// The lower triangle of A -= X X^T (the sums of tile_sub_xyt) by threads
// 0..127; what lies above the diagonal is not used afterwards.  FP32: the rows
// above 16 leave their upper half out.  FP64 (bound by its pipe: 64 cycles an
// instruction and warp): column c's 32 - c rows and column 32 - c's c rows
// share one warp, so 17 warp columns instead of 32.
__device__ __forceinline__ void tile_sub_sym(Tile<float>& A, const Tile<float>& X) {
  const int t = threadIdx.x;
  if (t >= 128) return;
  const int r = t >> 3, c0 = t & 7;
  float s0[2] = {0.0f, 0.0f}, s1[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int q = 0; q < kTile; q += 4) {
    float x0[4], x1[4];
    load16(&X[r][q], x0);
    load16(&X[r + 16][q], x1);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float y[4];
      load16(&X[c0 + 8 * u][q], y);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (u < 2) s0[u < 2 ? u : 0] = fmaf(x0[e], y[e], s0[u < 2 ? u : 0]);
        s1[u] = fmaf(x1[e], y[e], s1[u]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (u < 2) A[r][c0 + 8 * u] -= s0[u < 2 ? u : 0];
    A[r + 16][c0 + 8 * u] -= s1[u];
  }
}
// The same by 256 threads: the lower 128 take columns c0 and c0 + 8, the others
// c0 + 16 and c0 + 24 (of the rows from 16 on).
__device__ __forceinline__ void tile_sub_sym_half(Tile<float>& A, const Tile<float>& X) {
  const int t = threadIdx.x & 127, h = threadIdx.x >> 7;
  const int r = t >> 3, c0 = (t & 7) + 16 * h;
  float s0[2] = {0.0f, 0.0f}, s1[2] = {0.0f, 0.0f};
#pragma unroll
  for (int q = 0; q < kTile; q += 4) {
    float x0[4], x1[4];
    if (h == 0) load16(&X[r][q], x0);
    load16(&X[r + 16][q], x1);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float y[4];
      load16(&X[c0 + 8 * u][q], y);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (h == 0) s0[u] = fmaf(x0[e], y[e], s0[u]);
        s1[u] = fmaf(x1[e], y[e], s1[u]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (h == 0) A[r][c0 + 8 * u] -= s0[u];
    A[r + 16][c0 + 8 * u] -= s1[u];
  }
}
__device__ __forceinline__ void tile_sub_sym_half(Tile<double>&, const Tile<double>&) {}   // (FP64 rows keep two tiles)
__device__ __forceinline__ void tile_sub_sym(Tile<double>& A, const Tile<double>& X) {
  if (threadIdx.x >= 128) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = warp; c <= 16; c += 4) {
    const bool own = lane >= c;
    const int row = own ? lane : 32 - c + lane, col = own ? c : 32 - c;
    if (c == 16 && !own) continue;   // (column 16 is its own partner)
    double s = 0.0;
#pragma unroll 4
    for (int q = 0; q < kTile; q += 2) {
      double x[2], y[2];
      load16(&X[row][q], x);
      load16(&X[col][q], y);
      s = fma(x[0], y[0], s);
      s = fma(x[1], y[1], s);
    }
    A[row][col] -= s;
  }
}

// P = A Li^T for a lower triangular Li (a panel: Li = L_jj^-1) by kWarps warps
// (this one is the w-th): lane = row, warp w the columns 2 kWarps m + w and
// 2 kWarps m + 2 kWarps - 1 - w (an even split of the triangle).  The terms
// past a column's diagonal are zeros and are left out: the sums of tile_xyt
// in half its products.
template <int kWarps>
__device__ __forceinline__ int panel_col(int u, int w) { return kWarps * u + ((u & 1) ? kWarps - 1 - w : w); }

template <typename T, int kWarps>
__device__ __forceinline__ void tile_panel_sums(const Tile<T>& A, const Tile<T>& Li, int w, int lane,
                                                T (&s)[kTile / kWarps]) {
  constexpr int N = Vec16<T>::N, C = kTile / kWarps;
  int col[C];
#pragma unroll
  for (int u = 0; u < C; ++u) {
    col[u] = panel_col<kWarps>(u, w);
    s[u] = T(0);
  }
#pragma unroll
  for (int q = 0; q < kTile; q += N) {
    T x[N];
    load16(&A[lane][q], x);
#pragma unroll
    for (int u = 0; u < C; ++u) {
      if (q > kWarps * (u + 1) - 1) continue;   // (the column's range: col[u] < kWarps (u + 1))
      if (q <= col[u]) {
        T y[N];
        load16(&Li[col[u]][q], y);
#pragma unroll
        for (int e = 0; e < N; ++e) s[u] = fma(x[e], y[e], s[u]);
      }
    }
  }
}
// (P may not be A: other warps still read it)
template <typename T, int kWarps>
__device__ __forceinline__ void tile_panel(const Tile<T>& A, const Tile<T>& Li, Tile<T>& P, int w, int lane) {
  T s[kTile / kWarps];
  tile_panel_sums<T, kWarps>(A, Li, w, lane, s);
#pragma unroll
  for (int u = 0; u < kTile / kWarps; ++u) P[lane][panel_col<kWarps>(u, w)] = s[u];
}

// Factor the SPD tile D (lower triangle used; identity-padded) and write
// L^-1 to Dinv and its rows, as they are found, to Lg (unless null); called by
// the warps 0..3 of a CTA.  Columns are factored two at a time: the 2x2 pivot
// block gives both reciprocal square roots together (the second pivot is
// det / p0), no divisions.  Returns false (in one of the warps) when a pivot
// was not positive.  The two precisions split the work differently, with the
// same arithmetic per element.
constexpr int kPotrfBarrier = 1;   // named barriers 1 and 2: FP64 tile factorization (0 is __syncthreads)
constexpr int kQuadBarrier = 3;    // the four warps 0..3
constexpr int kAuxBarrier = 4;     // the four warps 4..7

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

// x > 0 without the FP64 pipe
__device__ __forceinline__ bool positive64(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7ff0000000000000LL;
}
// (one evaluation for both: an FP64 instruction costs the same for one lane)
__device__ __forceinline__ void rsqrt_two(double a, double b, double& ra, double& rb) {
  const double r = rsqrt((threadIdx.x & 1) ? b : a);
  ra = __shfl_sync(0xffffffffu, r, 0);
  rb = __shfl_sync(0xffffffffu, r, 1);
}

// Shared scratch of one tile factorization; `step` must be 0 before the first.
template <typename T>
struct PotrfBuf;
template <>
struct PotrfBuf<double> {
  double f[4][2][kTile];
  int step;
};
template <>
struct PotrfBuf<float> {
  alignas(16) float f[kTile / 2][2][kTile];   // the columns of L, pair by pair
  int step;                                     // pairs published so far
};

__device__ __forceinline__ void st_release_shared(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;\n" ::"r"(unsigned(__cvta_generic_to_shared(p))), "r"(v)
               : "memory");
}
__device__ __forceinline__ int ld_acquire_shared(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];\n"
               : "=r"(v)
               : "r"(unsigned(__cvta_generic_to_shared(p)))
               : "memory");
  return v;
}

// FP32: latency and one warp's issue slots.  Lane i of warp 0 keeps the
// columns 0..15 of row i in registers, lane i of warp 2 the columns 16..31,
// lane i of warp 1 column i of L^-1 (forward substitution against L).  Warp 0
// runs the first eight pairs without ever waiting for another, warp 2 applies
// each to its columns as it is published and then runs the last eight, warp 1
// follows one step behind.  A step's critical part goes through shuffles:
// the next pair's two columns are updated and its pivot block read first, the
// half's other columns (from the published ones, four to a load) fill the
// latency of the next square roots.  The waits (for `step`, which its owner
// always reaches) are bounded all the same.  In a loop 1,330 cycles; all 32
// columns in one warp took 2,630 (its issue slots), over four warps with a
// barrier a pair (the FP64 form) 4,400.  In the factorization's chain, where
// an SM runs it the second time only, 1.86 us (3,500 cycles).  Both halves run
// the same instructions (B at run time) and warp 2 applies the first half's
// pairs in a loop: 512 small systems, each a CTA's only factorization, 161 ->
// 148 us against a copy of the code per half.
__device__ __forceinline__ void potrf_half(float (&a)[kTile / 2], int B, PotrfBuf<float>& fb, int lane, bool& ok) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int H = kTile / 2;
  float p0 = __shfl_sync(FULL, a[0], B), p1 = __shfl_sync(FULL, a[0], B + 1), p2 = __shfl_sync(FULL, a[1], B + 1);
  // every column index is a compile-time constant, so a[] stays in registers
  static_for<0, H, 2>([&](auto hc) {
    constexpr int h = decltype(hc)::value;
    const int j = B + h, s = j / 2;
    const float det = fmaf(p0, p2, -(p1 * p1));
    const float r0 = rsqrtf(p0), rd = rsqrtf(det);
    const float l00 = p0 * r0;             // sqrt(p0)
    const float l10 = p1 * r0;
    const float r1 = l00 * rd;             // 1 / sqrt(det / p0)
    ok = ok && (p0 > 0.0f) && (det > 0.0f);
    const float li0 = lane > j ? a[h] * r0 : 0.0f;
    const float li1 = lane > j + 1 ? fmaf(-li0, l10, a[h + 1]) * r1 : 0.0f;
    // the diagonal's places carry the reciprocals for the inverse
    fb.f[s][0][lane] = lane == j ? r0 : li0;
    fb.f[s][1][lane] = lane == j + 1 ? r1 : li1;
    if constexpr (h + 2 < H) {
      const float c00 = __shfl_sync(FULL, li0, j + 2), c10 = __shfl_sync(FULL, li1, j + 2);
      const float c01 = __shfl_sync(FULL, li0, j + 3), c11 = __shfl_sync(FULL, li1, j + 3);
      a[h + 2] = fmaf(-li1, c10, fmaf(-li0, c00, a[h + 2]));
      a[h + 3] = fmaf(-li1, c11, fmaf(-li0, c01, a[h + 3]));
      p0 = __shfl_sync(FULL, a[h + 2], j + 2);
      p1 = __shfl_sync(FULL, a[h + 2], j + 3);
      p2 = __shfl_sync(FULL, a[h + 3], j + 3);
    }
    __syncwarp();
    if (lane == 0) st_release_shared(&fb.step, s + 1);
#pragma unroll
    for (int l = (h + 4) / 4 * 4; l < H; l += 4) {
      float c0[4], c1[4];
      load16(&fb.f[s][0][B + l], c0);
      load16(&fb.f[s][1][B + l], c1);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (l + e >= h + 4) a[l + e] = fmaf(-li1, c1[e], fmaf(-li0, c0[e], a[l + e]));
    }
  });
}

__device__ __forceinline__ bool tile_potrf_inverse(const Tile<float>& D, Tile<float>& Dinv, PotrfBuf<float>& fb,
                                                   float* __restrict__ Lg, int warp, int lane) {
  constexpr int H = kTile / 2;
  bool ok = true;
  auto wait_step = [&](int s) {
    for (int spin = 0; ld_acquire_shared(&fb.step) <= s && ok; ++spin) ok = spin < (1 << 20);
  };
  if (warp == 0 || warp == 2) {
    float a[H];
#pragma unroll
    for (int q = 0; q < H; q += 4) load16(&D[lane][(warp == 0 ? 0 : H) + q], a + q);
    if (warp == 2) {
#pragma unroll 1
      for (int s = 0; s < H / 2; ++s) {
        wait_step(s);
        const float li0 = fb.f[s][0][lane], li1 = fb.f[s][1][lane];
#pragma unroll
        for (int l = 0; l < H; l += 4) {
          float c0[4], c1[4];
          load16(&fb.f[s][0][H + l], c0);
          load16(&fb.f[s][1][H + l], c1);
#pragma unroll
          for (int e = 0; e < 4; ++e) a[l + e] = fmaf(-li1, c1[e], fmaf(-li0, c0[e], a[l + e]));
        }
      }
    }
    potrf_half(a, warp == 0 ? 0 : H, fb, lane, ok);
  } else if (warp == 1) {
    float x[kTile];
#pragma unroll
    for (int r = 0; r < kTile; ++r) x[r] = (r == lane) ? 1.0f : 0.0f;
    static_for<0, kTile / 2, 1>([&](auto sc) {
      constexpr int s = decltype(sc)::value, j = 2 * s;
      wait_step(s);
      const float r0 = fb.f[s][0][j], l10 = fb.f[s][0][j + 1], r1 = fb.f[s][1][j + 1];
      x[j] *= r0;
      x[j + 1] = fmaf(-l10, x[j], x[j + 1]) * r1;
      Dinv[j][lane] = x[j];
      Dinv[j + 1][lane] = x[j + 1];
      if (Lg) {
        Lg[j * kTile + lane] = x[j];
        Lg[(j + 1) * kTile + lane] = x[j + 1];
      }
#pragma unroll
      for (int l = (j + 2) / 4 * 4; l < kTile; l += 4) {
        float c0[4], c1[4];
        load16(&fb.f[s][0][l], c0);
        load16(&fb.f[s][1][l], c1);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (l + e >= j + 2) x[l + e] = fmaf(-c1[e], x[j + 1], fmaf(-c0[e], x[j], x[l + e]));
      }
    });
    __syncwarp();
    if (lane == 0) fb.step = 0;   // every pair is published and warp 2 waits for none of them
  }
  return ok;
}

// FP64: bound by its pipe (64 cycles an instruction and warp, whatever the
// lanes), so the work is spread over the four schedulers: the pair s =
// (2s, 2s + 1) belongs to warp s mod 4, lane t of which holds, for each of its
// columns l, the tile's entry (t, l) for t >= l and the inverse's entry (l, t)
// for t < l: a step's updates of both are the same FMAs with the step's two
// column vectors, so one instruction serves a column of the tile and a row of
// the inverse.  The pair's owner scales its two columns, publishes them (four
// buffers of two columns) and arrives at the step's barrier without waiting;
// the next pair's owner updates that pair first and publishes it before it
// catches up with its other columns.
__device__ __forceinline__ bool tile_potrf_inverse(const Tile<double>& D, Tile<double>& Dinv, PotrfBuf<double>& fb,
                                                   double* __restrict__ Lg, int warp, int lane) {
  using T = double;
  constexpr unsigned FULL = 0xffffffffu;
  bool ok = true;
  T v[8];   // columns 2 (warp + 4 p) + h at v[2 p + h]
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int l = 2 * (warp + 4 * p) + h;
      v[2 * p + h] = lane >= l ? D[lane][l] : T(0);
    }
  // step s's update of the warp's pair p
  auto update = [&](auto sc, auto pc) {
    constexpr int s = decltype(sc)::value, p = decltype(pc)::value;
    const T* f0 = fb.f[s & 3][0];
    const T* f1 = fb.f[s & 3][1];
    const int l = 2 * (warp + 4 * p);
    const T g0 = f0[lane], g1 = f1[lane];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const T c0 = f0[l + h], c1 = f1[l + h];
      const T a = fma(-g1, c1, fma(-g0, c0, v[2 * p + h]));
      if (lane >= l + h || lane <= 2 * s + 1) v[2 * p + h] = a;
    }
  };
  static_for<0, kTile / 2, 1>([&](auto sc) {
    constexpr int s = decltype(sc)::value, j = 2 * s, p = s >> 2;
    if (warp == (s & 3)) {   // the pair's owner: pivot, columns, publication
      const T a0 = v[2 * p], a1 = v[2 * p + 1];
      const T p0 = __shfl_sync(FULL, a0, j);
      const T p1 = __shfl_sync(FULL, a0, j + 1);
      const T p2 = __shfl_sync(FULL, a1, j + 1);
      const T det = fma(p0, p2, -(p1 * p1));
      T r0, rd;
      rsqrt_two(p0, det, r0, rd);
      const T f0 = lane == j ? r0 : a0 * r0;
      const T l00 = p0 * r0;             // sqrt(p0)
      const T l10 = __shfl_sync(FULL, f0, j + 1);   // p1 r0
      const T r1 = l00 * rd;             // 1 / sqrt(det / p0)
      ok = ok && positive64(p0) && positive64(det);
      const T f1 = lane == j + 1 ? r1 : fma(-f0, l10, a1) * r1;
      fb.f[s & 3][0][lane] = lane == j + 1 ? T(0) : f0;   // (row j of the inverse ends at j)
      fb.f[s & 3][1][lane] = f1;
      bar_arrive(kPotrfBarrier + (s & 1), 128);
      const T x0 = lane <= j ? f0 : T(0), x1 = lane <= j + 1 ? f1 : T(0);
      Dinv[j][lane] = x0;
      Dinv[j + 1][lane] = x1;
      if (Lg) {
        Lg[j * kTile + lane] = x0;
        Lg[(j + 1) * kTile + lane] = x1;
      }
      __syncwarp();
      // the other pairs: step s - 1 (left out below), then this step
      static_for<p + 1, 4, 1>([&](auto pc) {
        if constexpr (s > 0) update(std::integral_constant<int, (s > 0 ? s - 1 : 0)>{}, pc);
        update(sc, pc);
      });
    } else {
      bar_sync(kPotrfBarrier + (s & 1), 128);
      if (s + 1 < kTile / 2 && warp == ((s + 1) & 3)) {   // next: its pivot pair only
        constexpr int pn = s + 1 < kTile / 2 ? (s + 1) >> 2 : 3;
        update(sc, std::integral_constant<int, pn>{});
      } else {
        static_for<p, 4, 1>([&](auto pc) {
          constexpr int pp = decltype(pc)::value;
          if (pp > p || warp > (s & 3)) update(sc, pc);
        });
      }
    }
  });
  return ok;
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) k_chol_step(DevPlan d, int k) {
  __shared__ __align__(16) Tile<T> A, Li, Lj, D, Dinv;
  __shared__ T yk[kTile], tv[kTile];
  const int p = blockIdx.y;
  const LMState& st = d.state[p];
  if (!st.active || d.factor_flag[p]) return;
  const ProbInfo pi = d.prob[p];
  const int c = k + 1;
  const int Tn = pi.nt - c;           // tile rows c .. nt-1
  if (Tn <= 0) return;
  int i, j;
  if (k < 0) {                        // first launch: column 0 only
    if ((int)blockIdx.x >= Tn) return;
    i = blockIdx.x;
    j = 0;
  } else {
    const int lin = blockIdx.x;
    if (lin >= Tn * (Tn + 1) / 2) return;
    int ti = int((sqrtf(8.0f * float(lin) + 1.0f) - 1.0f) * 0.5f);
    while ((ti + 1) * (ti + 2) / 2 <= lin) ++ti;
    while (ti * (ti + 1) / 2 > lin) --ti;
    i = c + ti;
    j = c + (lin - ti * (ti + 1) / 2);
  }
  const int n = pi.n;
  T* S = tptr_mut<T>(d.S) + pi.s_off;
  T* b = tptr_mut<T>(d.b) + 6LL * pi.ext_begin;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // own tile and, for k >= 0, the column-k factors: all loads issued first
  TileFetch<T> fa, fi, fj, fd;
  if (i == j) fa.diag(S, n, i); else fa.rect(S, n, i, j);
  if (k >= 0) {
    fi.rect(S, n, i, k);
    fj.rect(S, n, j, k);
  }
  const bool need_d = (j == c && i != c);
  if (need_d) fd.diag(S, n, c);
  T ykv = T(0), bv = T(0);
  if (k >= 0 && tid < kTile) ykv = b[kTile * k + tid];   // y_k (tile k is full)
  if (j == c && tid < kTile && tid < tile_rows(n, i)) bv = b[kTile * i + tid];
  fa.store(A);
  if (k >= 0) {
    fi.store(Li);
    fj.store(Lj);
    if (tid < kTile) yk[tid] = ykv;
  }
  if (need_d) fd.store(D);
  __syncthreads();
  if (k >= 0) {
    if (i == j) tile_sub_sym(A, Li); else tile_sub_xyt<T>(A, Li, Lj);
    if (j == c && i != c) tile_sub_sym(D, Lj);
  }
  if (j == c && tid < kTile) {
    // b_i after column k: b_i - L_ik y_k
    T t = bv;
    if (k >= 0) {
#pragma unroll 8
      for (int q = 0; q < kTile; ++q) t -= Li[tid][q] * yk[q];
    }
    tv[tid] = t;
  }
  __syncthreads();
  if (j != c) {                       // trailing tile: write back
    const int mi = tile_rows(n, i), mj = tile_rows(n, j);
    for (int e = tid; e < kTile * kTile; e += blockDim.x) {
      const int r = e / kTile, q = e % kTile;
      if (r < mi && q < mj && (i != j || q <= r)) S[(long long)(kTile * i + r) * n + kTile * j + q] = A[r][q];
    }
    return;
  }
  // column c: factor the diagonal tile (own tile when i == c)
  __shared__ int ok_s;
  __shared__ PotrfBuf<T> fb;
  if (tid == 0) {
    ok_s = 1;
    fb.step = 0;
  }
  __syncthreads();
  if (warp < 4) {
    T* Lg = i == c ? tptr_mut<T>(d.Linv) + ((long long)p * d.max_nt + c) * kTile * kTile : nullptr;
    if (!tile_potrf_inverse(i == c ? A : D, Dinv, fb, Lg, warp, lane) && lane == 0) ok_s = 0;
  }
  __syncthreads();
  if (!ok_s) {
    if (tid == 0) d.factor_flag[p] = 1;
    return;
  }
  const int mi = tile_rows(n, i);
  if (i == c) {
    if (tid < mi) {
      T y = T(0);
#pragma unroll 8
      for (int q = 0; q < kTile; ++q) y += Dinv[tid][q] * tv[q];
      b[kTile * c + tid] = y;
    }
    return;
  }
  // i > c: L_ic = A_ic L_cc^-T, and the column-k part of the forward solve
  if (tid < mi) b[kTile * i + tid] = tv[tid];
  tile_panel<T, 8>(A, Dinv, Li, warp, lane);   // (Li is free again)
  __syncthreads();
  for (int r = warp; r < mi; r += 8) S[(long long)(kTile * i + r) * n + kTile * c + lane] = Li[r][lane];
}

// Dataflow factorization of one problem's reduced system in a single
// cooperative launch.  Every CTA owns a fixed set of tiles of the lower
// triangle (df_layout) and keeps them in shared memory for the whole
// factorization: row i's CTA its last ones, among them the diagonal tile (i, i)
// and the tile left of it, the others spread by work (j + 1 tasks for tile
// (i, j)).  A tile's tasks are its updates A_ij -= L_ik L_jk^T for
// k = 0 .. j-1, in that order, then its factorization (i == j, with the
// forward solve y_j = L_jj^-1 b_j) or its panel L_ij = A_ij L_jj^-T.  A
// finished factor or panel is written to global memory (L into S, L_jj^-1
// into Linv, y_j into b) and announced by storing the launch's epoch into
// the tile's flag with release semantics (y_j has its own, in the upper
// triangle of the flags); consumers poll the flags (acquire loads where one
// flag is waited for; relaxed ones, several in flight, and then a fence where a
// worker looks at all of its tiles) and read the data through L2.  Per
// element the arithmetic is exactly that of k_chol_step (same tile routines,
// same order of updates), so all schedules give the same bits.
//
// Without two CTAs per tile row each CTA runs, among its tiles whose next task
// has its inputs published, the one with the smallest (j, i), and applies up to
// df_batch consecutive ready updates of that tile with all of their loads in
// flight together.
//
// The critical path is the chain L_jj^-1 -> panel (j+1, j) -> last update of
// (j+1, j+1) -> its factor.  The chain task of a row does these in one go:
// warps 0..3 take the update and the factor, warps 4..7 meanwhile publish
// the panel (the next row's CTA then updates its own subdiagonal tile while
// this row is factored) and bring b_i up to date.  The rows of L_jj^-1 are
// stored as they are found, so the flag follows the last of them directly,
// before y_j.  With at least two CTAs per tile row (DevPlan::df_rows), row i's
// CTA owns nothing but the row's last tiles (df_row_tiles) and runs a fixed
// program instead of that scheduler: the updates of all of them column by
// column, then the panel (i, i-2) with its updates, then the chain task, so
// that the row is always waiting for L_{i-1,i-1}^-1 when it comes.  Scheduled
// tile by tile, every second row was late for it by an update of its
// diagonal tile and ran its panel, that update and its factor as three tasks
// (7.5 us a row instead of 4.1).  With at least four CTAs per row (FP32), a
// second CTA keeps the three columns left of those in the same way
// (df_helpers): panels that wait their turn in a worker's queue are then needed
// several chain steps later instead of one.  The other CTAs are workers
// (worker_program).
//
// Every wait is bounded: a CTA that sees nothing ready for
// DevPlan::df_spin_limit polls records a timeout and leaves; a failed pivot
// or a timeout raises the abort word, which every waiting CTA checks.
constexpr int kDfThreads = 256;

template <typename T>
__host__ __device__ constexpr int df_batch() { return 2; }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// A relaxed poll: several of one thread are in flight together (acquire loads
// wait for one another); a fence must follow before the data is read.
__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Tile loads through L2 (data another CTA published in this launch).
template <typename T>
__device__ __forceinline__ void fetch_rect_cg(TileFetch<T>& f, const T* S, int n, int ti, int tj) {
  const int mi = tile_rows(n, ti), mj = tile_rows(n, tj);
#pragma unroll
  for (int u = 0; u < kPerThread; ++u) {
    const int e = threadIdx.x + u * kCholThreads, r = e / kTile, c = e % kTile;
    f.v[u] = (r < mi && c < mj) ? __ldcg(S + (long long)(kTile * ti + r) * n + kTile * tj + c) : T(0);
  }
}

// The tile (ti, tj) left of the diagonal (all 32 columns) through L2 by the
// threads t = 0 .. 127 of a thread group.
template <typename T>
struct HalfFetch {
  T v[kTile * kTile / 128];
  __device__ __forceinline__ void load(const T* S, int n, int ti, int tj, int t) {
    const int mi = tile_rows(n, ti), r0 = t >> 5, c = t & 31;
    const T* p = S + (long long)(kTile * ti + r0) * n + kTile * tj + c;
#pragma unroll
    for (int u = 0; u < kTile / 4; ++u) v[u] = r0 + 4 * u < mi ? __ldcg(p + (long long)(4 * u) * n) : T(0);
  }
  __device__ __forceinline__ void store(Tile<T>& tile, int t) const {
#pragma unroll
    for (int u = 0; u < kTile / 4; ++u) tile[(t >> 5) + 4 * u][t & 31] = v[u];
  }
};

// A contiguous 32x32 tile (an L_jj^-1) through L2, 16 bytes a load, by the
// threads t = 0 .. kThreads - 1 of a thread group.
template <typename T, int kThreads>
struct InvFetch {
  static constexpr int N = Vec16<T>::N, kVecs = kTile * kTile / N / kThreads;
  typename Vec16<T>::V v[kVecs];
  __device__ __forceinline__ void load(const T* Li, int t) {
#pragma unroll
    for (int u = 0; u < kVecs; ++u)
      v[u] = __ldcg(reinterpret_cast<const typename Vec16<T>::V*>(Li) + t + u * kThreads);
  }
  __device__ __forceinline__ void store(Tile<T>& tile, int t) const {
#pragma unroll
    for (int u = 0; u < kVecs; ++u) {
      const int e = (t + u * kThreads) * N;
      *reinterpret_cast<typename Vec16<T>::V*>(&tile[e / kTile][e % kTile]) = v[u];
    }
  }
};

template <typename T>
size_t df_smem_bytes(int max_own) {
  return sizeof(Tile<T>) * size_t(max_own + 2 * df_batch<T>() + 1) +
         sizeof(T) * size_t(max_own) * kTile + sizeof(int) * size_t(5 * max_own + 8);
}

template <typename T>
__global__ void __launch_bounds__(kDfThreads, 1) k_chol_dataflow(DevPlan d) {
  constexpr int NB = df_batch<T>();
  enum { kIdle = 0, kUpdate = 1, kFinish = 2, kChain = 3, kExit = 4 };
  extern __shared__ __align__(16) unsigned char df_raw[];
  __shared__ T yv[NB][kTile];
  __shared__ PotrfBuf<T> fb;
  __shared__ int s_sel, s_cnt, s_mode, s_ok;
  const int p = 0;
  const ProbInfo pi = d.prob[p];
  const int n = pi.n, nt = pi.nt;
  const int ob = d.df_own_off[blockIdx.x], nown = d.df_own_off[blockIdx.x + 1] - ob;
  const int mo = d.df_max_own;
  Tile<T>* A = reinterpret_cast<Tile<T>*>(df_raw);   // [mo] owned tiles
  Tile<T>* W = A + mo;                                // [2 * NB] fetched L tiles
  Tile<T>& Dinv = W[2 * NB];
  T* bown = reinterpret_cast<T*>(W + 2 * NB + 1);     // [mo][kTile] rhs of owned diagonal tiles
  int* ti_s = reinterpret_cast<int*>(bown + size_t(mo) * kTile);
  int* tj_s = ti_s + mo;
  int* kt_s = tj_s + mo;       // next update step of each owned tile (j: factor/panel; j+1: done)
  int* rd_s = kt_s + mo;       // ready tasks found by the last poll
  int* pr_s = rd_s + mo;       // tile (i, i-1): local index of (i, i); otherwise -1
  T* S = tptr_mut<T>(d.S) + pi.s_off;
  T* b = tptr_mut<T>(d.b) + 6LL * pi.ext_begin;
  T* Lg = tptr_mut<T>(d.Linv) + (long long)p * d.max_nt * kTile * kTile;
  unsigned* flags = d.df_flags;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned epoch = *reinterpret_cast<volatile unsigned*>(d.df_sync) + 1u;

  // optional timeline (thread 0): per task its wait start, selection, end
  unsigned long long* tr = d.df_trace ? d.df_trace + size_t(blockIdx.x) * kDfTraceCap * 4 : nullptr;
  // y_k's flag (row 0 of the upper triangle; nobody waits for the last y)
  auto y_flag = [&](int kk) { return flags + kk + 1; };
  // L_ii^-1 of row i is out (warps 0..3 stored its rows): announce it, then
  // form and announce y_i = L_ii^-1 b_i; false (after raising the abort word)
  // on a bad pivot
  auto finish_diag = [&](int t, int i) -> bool {
    __syncthreads();
    if (s_ok <= 0) {
      if (tid == 0 && s_ok == 0) {
        d.factor_flag[p] = 1;
        __threadfence();
        atomicExch(d.df_sync + 2, epoch);
      }
      return false;
    }
    if (tid == 0) st_release_u32(flags + (long long)i * nt + i, epoch);
    if (warp == 1) {
      T y = T(0);
#pragma unroll 8
      for (int q = 0; q < kTile; ++q) y += Dinv[lane][q] * bown[t * kTile + q];
      if (lane < tile_rows(n, i)) b[kTile * i + lane] = y;
      __syncwarp();
      if (lane == 0 && i + 1 < nt) st_release_u32(y_flag(i), epoch);
    }
    if (tid == 0) kt_s[t] = i + 1;
    return true;
  };

  // W[0] = the panel L_ij = A_ij L_jj^-T (L_jj^-1 is published); ends with a barrier
  auto panel_of = [&](const Tile<T>& Aij, int j) {
    InvFetch<T, kDfThreads> f;
    f.load(Lg + (long long)j * kTile * kTile, tid);
    f.store(Dinv, tid);
    __syncthreads();
    tile_panel<T, 8>(Aij, Dinv, W[0], warp, lane);
    __syncthreads();
  };
  // the rows of the panel W[0] into S, by `warps` warps (this one is the w-th)
  auto publish_panel = [&](int i, int j, int w, int warps) {
    const int mi = tile_rows(n, i);
    T* const Sij = S + (long long)kTile * i * n + kTile * j;
    for (int r = w; r < mi; r += warps) Sij[(long long)r * n + lane] = W[0][r][lane];
  };
  // one warp waits for the flags f[0 .. cnt) (one per lane; null: none);
  // false when the launch is aborted or the limit ran out
  auto wait_flag = [&](const unsigned* f) -> bool {
    long long spin = 0;
    for (;;) {
      if (__all_sync(0xffffffffu, f == nullptr || ld_acquire_u32(f) == epoch)) return true;
      ++spin;
      int stop = 0;
      if (lane == 0 && (spin & 15) == 0) stop = ld_acquire_u32(d.df_sync + 2) == epoch;
      if (lane == 0 && !stop && spin > d.df_spin_limit) {
        d.factor_flag[p] = 2;   // timed out
        __threadfence();
        atomicExch(d.df_sync + 2, epoch);
        stop = 1;
      }
      if (__shfl_sync(0xffffffffu, stop, 0)) return false;
    }
  };
  // bown[t] -= L yv[0] for a tile L of row i (one warp)
  auto rhs_sub = [&](int t, const Tile<T>& L) {
    T tv = bown[t * kTile + lane];
#pragma unroll 8
    for (int q = 0; q < kTile; ++q) tv -= L[lane][q] * yv[0][q];
    bown[t * kTile + lane] = tv;
  };
  // bown[t] -= L y_k once y_k is out (one warp); false when aborted
  auto row_rhs = [&](int t, const Tile<T>& L, int kk) -> bool {
    if (!wait_flag(lane == 0 ? y_flag(kk) : nullptr)) return false;
    yv[0][lane] = __ldcg(b + kTile * kk + lane);
    __syncwarp();
    rhs_sub(t, L);
    __syncwarp();
    return true;
  };
  // the chain task of row i (tile t = (i, i-1), td = (i, i)); false when it
  // failed or the launch is aborted
  auto chain_task = [&](int t, int td, int i) -> bool {
    const int j = i - 1;
    panel_of(A[t], j);
    if (warp < 4) {
      tile_sub_sym(A[td], W[0]);
      bar_sync(kQuadBarrier, 128);
      if (!tile_potrf_inverse(A[td], Dinv, fb, Lg + (long long)i * kTile * kTile, warp, lane) && lane == 0)
        s_ok = 0;
    } else {
      publish_panel(i, j, warp - 4, 4);
      bar_sync(kAuxBarrier, 128);
      if (tid == 128) st_release_u32(flags + (long long)i * nt + j, epoch);
      if (warp == 5 && !row_rhs(td, W[0], j) && lane == 0) s_ok = -1;
    }
    return finish_diag(td, i);
  };
  // every thread waits while warp 0 polls (one flag per lane)
  auto cta_wait = [&](const unsigned* f) -> bool {
    if (warp == 0) {
      const bool ok = wait_flag(f);
      if (lane == 0) s_mode = ok ? 1 : 0;
    }
    __syncthreads();
    const bool ok = s_mode != 0;
    __syncthreads();
    return ok;
  };
  // the fixed program of row i's own CTA: its tiles are (i, i-2), (i, i-1),
  // (i, i) (the last `nown` of them).  The chain task runs once per CTA, so its
  // instructions would come from L2 while every later row waits: it is run
  // through once on scratch tiles first, from the same code.
  int rp_n = 0;
  unsigned long long rp_wait = 0, rp_sel = 0;
  auto note_wait = [&] { if (tr && tid == 0) rp_wait = global_ns(); };
  auto note_start = [&] { if (tr && tid == 0) rp_sel = global_ns(); };
  auto note_end = [&](int mode, int j, int kk) {
    if (!tr || tid != 0 || rp_n >= kDfTraceCap) return;
    unsigned long long* e = tr + 4 * rp_n++;
    e[0] = (unsigned long long)mode << 56 | (unsigned long long)blockIdx.x << 40 | (unsigned long long)j << 24 |
           (unsigned long long)kk << 8 | 1ull;
    e[1] = rp_wait;
    e[2] = rp_sel;
    e[3] = global_ns();
  };
  auto row_chain = [&](int i, int t1, int td, bool real) {
    if (i > 0) {
      if (real) {
        panel_of(A[t1], i - 1);
      } else {
        tile_panel<T, 8>(W[1], W[2], W[0], warp, lane);
        __syncthreads();
      }
    }
    if (warp < 4) {
      Tile<T>& Di = real ? A[td] : W[3];
      if (i > 0) tile_sub_sym(Di, W[0]);
      bar_sync(kQuadBarrier, 128);
      if (!tile_potrf_inverse(Di, Dinv, fb, real ? Lg + (long long)i * kTile * kTile : nullptr, warp, lane) &&
          lane == 0 && real)
        s_ok = 0;
    } else if (i > 0 && real) {
      publish_panel(i, i - 1, warp - 4, 4);
      bar_sync(kAuxBarrier, 128);
      if (tid == 128) st_release_u32(flags + (long long)i * nt + i - 1, epoch);
      if (warp == 5 && !row_rhs(td, W[0], i - 1) && lane == 0) s_ok = -1;
    }
    if (real)
      finish_diag(td, i);
    else
      __syncthreads();
  };
  auto row_steps = [&](int i) -> bool {
    const int td = nown - 1, t1 = nown - 2, t2 = nown - 3;   // (negative: none)
    const int steps = t2 >= 0 ? i - 2 : i - 1;
    for (int kk = 0; kk < steps; ++kk) {   // column kk into every tile of the row
      note_wait();
      const unsigned* f = nullptr;
      if (lane == 0) f = flags + (long long)i * nt + kk;
      if (lane == 1) f = flags + (long long)(i - 1) * nt + kk;
      if (lane == 2 && t2 >= 0) f = flags + (long long)(i - 2) * nt + kk;
      if (lane == 3) f = y_flag(kk);
      if (!cta_wait(f)) return false;
      note_start();
      {
        TileFetch<T> f0, f1, f2;
        fetch_rect_cg<T>(f0, S, n, i, kk);
        fetch_rect_cg<T>(f1, S, n, i - 1, kk);
        if (t2 >= 0) fetch_rect_cg<T>(f2, S, n, i - 2, kk);
        if (warp == 0) yv[0][lane] = __ldcg(b + kTile * kk + lane);
        f0.store(W[0]);
        f1.store(W[1]);
        if (t2 >= 0) f2.store(W[2]);
      }
      __syncthreads();
      if (t2 >= 0) {
        tile_sub_xyt_t<T>(A[warp < 4 ? t2 : t1], W[0], W[warp < 4 ? 2 : 1], tid & 127);
        tile_sub_sym_half(A[td], W[0]);
      } else if (warp < 4) {
        tile_sub_sym(A[td], W[0]);
      } else {
        tile_sub_xyt_t<T>(A[t1], W[0], W[1], tid - 128);
      }
      if (warp == 7) rhs_sub(td, W[0]);
      __syncthreads();
      note_end(kUpdate, i, kk);
    }
    if (t2 >= 0) {   // the panel (i, i-2), then its column into the other two
      const int j = i - 2;
      note_wait();
      if (!cta_wait(lane == 0 ? flags + (long long)j * nt + j : nullptr)) return false;
      note_start();
      panel_of(A[t2], j);
      bool ok = true;
      if (warp < 4) {
        tile_sub_sym(A[td], W[0]);
      } else {
        publish_panel(i, j, warp - 4, 4);
        bar_sync(kAuxBarrier, 128);
        if (tid == 128) st_release_u32(flags + (long long)i * nt + j, epoch);
        if (warp == 5) ok = row_rhs(td, W[0], j);
        if (warp == 6) ok = wait_flag(lane == 0 ? flags + (long long)(i - 1) * nt + j : nullptr);
      }
      if (!ok && lane == 0) s_ok = -1;
      __syncthreads();
      if (s_ok < 0) return false;
      TileFetch<T> f1;
      fetch_rect_cg<T>(f1, S, n, i - 1, j);
      f1.store(W[1]);
      __syncthreads();
      tile_sub_xyt<T>(A[t1], W[0], W[1]);
      __syncthreads();
      note_end(kFinish, j, j);
    }
    note_wait();
    if (t1 >= 0 && !cta_wait(lane == 0 ? flags + (long long)(i - 1) * nt + i - 1 : nullptr)) return false;
    note_start();
    return true;
  };
  // the program of row i's second CTA (DevPlan::df_helpers): its tiles are
  // the (up to three) columns left of the first CTA's, c0 .. c0 + nown - 1,
  // updated together column by column, then their panels in order, each
  // taken into the tiles right of it as soon as it is out
  auto helper_program = [&](int i) -> bool {
    const int c0 = i - 2 - nown;
    for (int kk = 0; kk < c0; ++kk) {
      const unsigned* f = nullptr;
      if (lane == 0) f = flags + (long long)i * nt + kk;
      if (lane >= 1 && lane <= nown) f = flags + (long long)(c0 + lane - 1) * nt + kk;
      if (!cta_wait(f)) return false;
      {
        TileFetch<T> f0, f1, f2, f3;
        fetch_rect_cg<T>(f0, S, n, i, kk);
        fetch_rect_cg<T>(f1, S, n, c0, kk);
        if (nown > 1) fetch_rect_cg<T>(f2, S, n, c0 + 1, kk);
        if (nown > 2) fetch_rect_cg<T>(f3, S, n, c0 + 2, kk);
        f0.store(W[0]);
        f1.store(W[1]);
        if (nown > 1) f2.store(W[2]);
        if (nown > 2) f3.store(W[3]);
      }
      __syncthreads();
      for (int t = tid >> 7; t < nown; t += 2) tile_sub_xyt_t<T>(A[t], W[0], W[1 + t], tid & 127);
      __syncthreads();
    }
    for (int u = 0; u < nown; ++u) {
      const int j = c0 + u;
      if (!cta_wait(lane == 0 ? flags + (long long)j * nt + j : nullptr)) return false;
      panel_of(A[u], j);
      publish_panel(i, j, warp, 8);
      __syncthreads();
      if (tid == 128) st_release_u32(flags + (long long)i * nt + j, epoch);
      if (u + 1 < nown) {
        const int m = nown - u - 1;   // tiles right of it
        if (!cta_wait(lane >= 1 && lane <= m ? flags + (long long)(j + lane) * nt + j : nullptr)) return false;
        TileFetch<T> f1, f2;
        fetch_rect_cg<T>(f1, S, n, j + 1, j);
        if (m > 1) fetch_rect_cg<T>(f2, S, n, j + 2, j);
        f1.store(W[1]);
        if (m > 1) f2.store(W[2]);
        __syncthreads();
        const int t = tid >> 7;
        if (t < m) tile_sub_xyt_t<T>(A[u + 1 + t], W[0], W[1 + t], tid & 127);
        __syncthreads();
      }
    }
    return true;
  };
  // a worker CTA beside row CTAs (df_rows): its two halves of four warps are
  // workers of their own, half g with the tiles t = g (mod 2), so that one's
  // loads and waits overlap the other's products.  Lane m of the half's first
  // warp keeps its m-th tile's state (at most 32 tiles) and polls its flags;
  // the ready tile with the smallest (j, i) is taken, up to four updates at a
  // time with the next one's loads in flight, or its panel.
  auto worker_program = [&] {
    const int g = tid >> 7, gt = tid & 127, gw = warp & 3, bar = kQuadBarrier + g;
    Tile<T>& X = W[2 * g];
    Tile<T>& Y = W[2 * g + 1];
    __shared__ int4 s_task[2];   // (tile, first column, count or 0: panel, 0 leave / 1 go / 2 wait)
    int my_t = -1, my_i = 0, my_j = 0, my_k = 0;
    if (gw == 0 && 2 * lane + g < nown) {
      my_t = 2 * lane + g;
      my_i = ti_s[my_t];
      my_j = tj_s[my_t];
    }
    int left = (nown - g + 1) / 2, rp_n = 0;
    long long spin = 0;
    unsigned long long t_wait = 0, t_sel = 0;
    if (tr && gt == 0) t_wait = global_ns();
    while (left > 0) {
      if (gw == 0) {
        int c = 0, ready = 0;   // c updates ready, or the panel
        if (my_t >= 0 && my_k < my_j) {
          unsigned fi[4], fj[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            fi[u] = my_k + u < my_j ? ld_relaxed_u32(flags + (long long)my_i * nt + my_k + u) : 0u;
            fj[u] = my_k + u < my_j ? ld_relaxed_u32(flags + (long long)my_j * nt + my_k + u) : 0u;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (c == u && my_k + u < my_j && fi[u] == epoch && fj[u] == epoch) c = u + 1;
          ready = c > 0;
        } else if (my_t >= 0 && my_k == my_j) {
          ready = ld_relaxed_u32(flags + (long long)my_j * nt + my_j) == epoch;
        }
        const unsigned any = __ballot_sync(0xffffffffu, ready);   // (lanes are in (j, i) order)
        if (any != 0) {
          if (lane == __ffs(any) - 1) {
            __threadfence();   // acquire what the polled flags announce
            s_task[g] = make_int4(my_t, my_k, c, 1);
            my_k += c > 0 ? c : 1;
          }
        } else {
          ++spin;
          if (lane == 0) {
            int go = 2;
            if ((spin & 15) == 0 && ld_acquire_u32(d.df_sync + 2) == epoch) {
              go = 0;
            } else if (spin > d.df_spin_limit) {
              d.factor_flag[p] = 2;   // timed out
              __threadfence();
              atomicExch(d.df_sync + 2, epoch);
              go = 0;
            }
            s_task[g] = make_int4(0, 0, 0, go);
          }
        }
      }
      bar_sync(bar, 128);
      const int4 task = s_task[g];
      if (task.w == 0) return;
      if (task.w == 2) {
        bar_sync(bar, 128);
        continue;
      }
      if (tr && gt == 0) t_sel = global_ns();
      const int t = task.x, i = ti_s[t], j = tj_s[t];
      if (task.z > 0) {
        HalfFetch<T> fx, fy;
        fx.load(S, n, i, task.y, gt);
        fy.load(S, n, j, task.y, gt);
        for (int u = 0; u < task.z; ++u) {
          fx.store(X, gt);
          fy.store(Y, gt);
          bar_sync(bar, 128);
          if (u + 1 < task.z) {
            fx.load(S, n, i, task.y + u + 1, gt);
            fy.load(S, n, j, task.y + u + 1, gt);
          }
          tile_sub_xyt_t<T>(A[t], X, Y, gt);
          bar_sync(bar, 128);
        }
      } else {
        InvFetch<T, 128> f;
        f.load(Lg + (long long)j * kTile * kTile, gt);
        f.store(X, gt);
        bar_sync(bar, 128);
        tile_panel<T, 4>(A[t], X, Y, gw, lane);
        bar_sync(bar, 128);
        const int mi = tile_rows(n, i);
        T* const Sij = S + (long long)kTile * i * n + kTile * j;
        for (int r = gw; r < mi; r += 4) Sij[(long long)r * n + lane] = Y[r][lane];
        bar_sync(bar, 128);
        if (gt == 96) st_release_u32(flags + (long long)i * nt + j, epoch);
        --left;
      }
      if (tr && gt == 0 && rp_n < kDfTraceCap / 2) {
        unsigned long long* e = tr + 4 * (2 * rp_n++ + g);
        e[0] = (unsigned long long)(task.z > 0 ? kUpdate : kFinish) << 56 | (unsigned long long)i << 40 |
               (unsigned long long)j << 24 | (unsigned long long)task.y << 8 | (unsigned long long)task.z;
        e[1] = t_wait;
        e[2] = t_sel;
        e[3] = t_wait = global_ns();
      }
    }
  };
  auto row_program = [&](int i) {
    for (int pass = i > 0 ? 0 : 1; pass < 2; ++pass) {   // (row 0 starts at once)
      if (pass == 1 && !row_steps(i)) return;
      row_chain(i, nown - 2, nown - 1, pass == 1);
    }
    note_end(kChain, i - 1, i - 1);
  };

  if (tid == 0) {
    s_ok = 1;
    fb.step = 0;
  }
  const LMState& st = d.state[p];
  const bool run = st.active && !d.factor_flag[p];
  if (run) {
    if (tr)   // (a launch with nothing to do keeps the last one's)
      for (int e = tid; e < 4 * kDfTraceCap; e += blockDim.x) tr[e] = 0ull;
    for (int t = tid; t < nown; t += blockDim.x) {
      const int2 tl = d.df_own[ob + t];
      ti_s[t] = tl.x;
      tj_s[t] = tl.y;
      kt_s[t] = 0;
    }
    __syncthreads();
    for (int t = tid; t < nown; t += blockDim.x) {
      int pr = -1;
      if (tj_s[t] == ti_s[t] - 1)
        for (int u = 0; u < nown; ++u)
          if (ti_s[u] == ti_s[t] && tj_s[u] == ti_s[t]) pr = u;
      pr_s[t] = pr;
    }
    for (int t0 = 0; t0 < nown; t0 += 4) {      // owned tiles and rhs, four tiles in flight
      TileFetch<T> f[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (t0 + u < nown) {
          const int i = ti_s[t0 + u], j = tj_s[t0 + u];
          if (i == j) f[u].diag(S, n, i); else f[u].rect(S, n, i, j);
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (t0 + u < nown) {
          const int t = t0 + u, i = ti_s[t];
          f[u].store(A[t]);
          if (i == tj_s[t] && tid < kTile) bown[t * kTile + tid] = tid < tile_rows(n, i) ? b[kTile * i + tid] : T(0);
        }
    }
  }
  __syncthreads();
  const int bx = int(blockIdx.x);
  const bool row_cta = bx < d.df_rows + d.df_helpers;
  if (run && bx < d.df_rows)
    row_program(bx);
  else if (run && row_cta && nown > 0)
    helper_program(bx - d.df_rows);
  else if (run && d.df_rows > 0 && nown > 0)
    worker_program();
  int ndone = run && d.df_rows == 0 ? 0 : nown;   // (without row CTAs: the scheduler below)
  long long idle = 0;
  unsigned long long tr_wait = 0, tr_sel = 0, tr_meta = 0;
  int tr_n = 0;
  bool tr_open = false;
  if (tr && tid == 0) tr_wait = global_ns();
  while (ndone < nown) {
    if (tr && tid == 0 && tr_open) {
      const unsigned long long now = global_ns();
      if (tr_n < kDfTraceCap) {
        unsigned long long* e = tr + 4 * tr_n;
        e[0] = tr_meta;
        e[1] = tr_wait;
        e[2] = tr_sel;
        e[3] = now;
      }
      ++tr_n;
      tr_open = false;
      tr_wait = now;
    }
    // poll: for each owned tile, how many of its next tasks have their inputs
    for (int t = tid; t < nown; t += blockDim.x) {
      const int i = ti_s[t], j = tj_s[t], k = kt_s[t];
      int c = 0;
      if (k < j) {
        unsigned fi[NB], fj[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
          fi[u] = (k + u < j) ? ld_acquire_u32(flags + (long long)i * nt + k + u) : 0u;
          fj[u] = (k + u < j) ? ld_acquire_u32(i != j ? flags + (long long)j * nt + k + u : y_flag(k + u)) : epoch;
        }
#pragma unroll
        for (int u = 0; u < NB; ++u)
          if (c == u && k + u < j && fi[u] == epoch && fj[u] == epoch) c = u + 1;
      } else if (k == j) {
        c = (i == j || ld_acquire_u32(flags + (long long)j * nt + j) == epoch) ? 1 : 0;
      }
      rd_s[t] = c;
    }
    __syncthreads();
    if (tid == 0) {
      int sel = -1, cnt = 0, mode = kIdle;
      for (int t = 0; t < nown; ++t) {
        if (rd_s[t] > 0) {
          sel = t;
          cnt = rd_s[t];
          mode = kt_s[t] < tj_s[t] ? kUpdate : kFinish;
          // a subdiagonal panel with its diagonal tile one update short
          if (mode == kFinish && pr_s[t] >= 0 && kt_s[pr_s[t]] == ti_s[t] - 1) mode = kChain;
          break;
        }
      }
      // nothing left but the chain task: wait here for the one flag it
      // needs, with the bounds of the general loop
      if (sel < 0 && nown - ndone == 2) {
        for (int t = 0; t < nown; ++t)
          if (pr_s[t] >= 0 && kt_s[t] == tj_s[t] && kt_s[pr_s[t]] == ti_s[t] - 1) {
            const unsigned* fl = flags + (long long)tj_s[t] * nt + tj_s[t];
            while (idle <= d.df_spin_limit) {
              if (ld_acquire_u32(fl) == epoch) {
                sel = t;
                cnt = 1;
                mode = kChain;
                break;
              }
              if ((++idle & 15) == 0 && ld_acquire_u32(d.df_sync + 2) == epoch) {
                mode = kExit;
                break;
              }
            }
          }
      }
      if (sel < 0 && mode != kExit) {
        // the abort word is read every 16th idle round, the limit counted always
        if ((++idle & 15) == 0 && ld_acquire_u32(d.df_sync + 2) == epoch) {
          mode = kExit;
        } else if (idle > d.df_spin_limit) {
          d.factor_flag[p] = 2;                       // timed out
          __threadfence();
          atomicExch(d.df_sync + 2, epoch);
          mode = kExit;
        }
      }
      s_sel = sel;
      s_cnt = cnt;
      s_mode = mode;
      if (tr && sel >= 0) {
        tr_sel = global_ns();
        tr_meta = (unsigned long long)mode << 56 | (unsigned long long)ti_s[sel] << 40 |
                  (unsigned long long)tj_s[sel] << 24 | (unsigned long long)kt_s[sel] << 8 |
                  (unsigned long long)cnt;
        tr_open = true;
      }
    }
    __syncthreads();
    const int mode = s_mode, t = s_sel, cnt = s_cnt;
    if (mode == kExit) break;
    if (mode == kIdle) continue;
    const int i = ti_s[t], j = tj_s[t], k0 = kt_s[t];
    if (mode == kUpdate) {
      // cnt consecutive updates from columns k0 .. k0+cnt-1
      TileFetch<T> fi[NB], fj[NB];
      T yr[NB];
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        if (u < cnt) {
          fetch_rect_cg<T>(fi[u], S, n, i, k0 + u);
          if (i != j) fetch_rect_cg<T>(fj[u], S, n, j, k0 + u);
          if (i == j && tid < kTile) yr[u] = __ldcg(b + kTile * (k0 + u) + tid);
        }
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {
        if (u < cnt) {
          fi[u].store(W[2 * u]);
          if (i != j) fj[u].store(W[2 * u + 1]);
          if (i == j && tid < kTile) yv[u][tid] = yr[u];
        }
      }
      __syncthreads();
      for (int u = 0; u < cnt; ++u) {
        if (i == j) tile_sub_sym(A[t], W[2 * u]); else tile_sub_xyt<T>(A[t], W[2 * u], W[2 * u + 1]);
        if (i == j && tid < kTile) {
          T tv = bown[t * kTile + tid];
#pragma unroll 8
          for (int q = 0; q < kTile; ++q) tv -= W[2 * u][tid][q] * yv[u][q];
          bown[t * kTile + tid] = tv;
        }
      }
      __syncthreads();
      if (tid == 0) kt_s[t] = k0 + cnt;
      __syncthreads();
      continue;
    }
    if (i == j) {                          // factor a diagonal tile
      if (warp < 4 &&
          !tile_potrf_inverse(A[t], Dinv, fb, Lg + (long long)i * kTile * kTile, warp, lane) && lane == 0)
        s_ok = 0;
      if (!finish_diag(t, i)) break;
      ++ndone;
      __syncthreads();
      continue;
    }
    if (mode == kChain) {
      if (!chain_task(t, pr_s[t], i)) break;
      ++ndone;
    } else {
      panel_of(A[t], j);
      publish_panel(i, j, warp, 8);
      __syncthreads();
      if (tid == 0) st_release_u32(flags + (long long)i * nt + j, epoch);
    }
    if (tid == 0) kt_s[t] = j + 1;
    ++ndone;
    __syncthreads();
  }
  if (tr && tid == 0 && tr_open && tr_n < kDfTraceCap) {
    unsigned long long* e = tr + 4 * tr_n;
    e[0] = tr_meta;
    e[1] = tr_wait;
    e[2] = tr_sel;
    e[3] = global_ns();
  }
  // the last CTA to finish opens the next epoch
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(d.df_sync + 1, 1u);
    if (prev == gridDim.x - 1) {
      d.df_sync[1] = 0u;
      __threadfence();
      atomicAdd(d.df_sync, 1u);
    }
  }
}

// Backward solve L^T delta = y in one launch per batch.  Problems with more
// than kSolveSmallTiles tile rows get a cluster of kSolveRanks CTAs, the
// others one CTA (R = 1).  Rank q owns the tile rows t = q (mod R) of y in
// shared memory.  Step j (nt-1 down to 0): warp 7 of the owner of row j
// forms delta_j = L_jj^-T y_j (y_j is final: its last update came from this
// same CTA at step j+1) and stores it into every rank's shared memory; after
// a cluster barrier every rank subtracts L_ji^T delta_j from its rows i < j,
// warp w taking rows q + R*(w + 8u), reading row block j of L coalesced
// along the row with the next step's loads already in flight.  The barrier
// arrives relaxed (it must not wait for those loads); the delta stores are
// ordered by a cluster-scope fence in the storing warp.
constexpr int kSolveRanks = 8;
constexpr int kSolveSmallTiles = 8;
constexpr int kSolveOwnerWarp = 7;

__device__ __forceinline__ void cluster_arrive_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void fence_cluster() {
  asm volatile("fence.acq_rel.cluster;\n" ::: "memory");
}

template <typename T, int R>
__device__ __forceinline__ void chol_solve_body(const DevPlan& d, int q) {
  constexpr int kRows = R == 1 ? kSolveSmallTiles : (6 * 2048 / kTile + R - 1) / R;
  __shared__ T ys[kRows][kTile];
  __shared__ T xb[2][kTile];
  const int p = blockIdx.y;
  const LMState& st = d.state[p];
  if (!st.active || d.factor_flag[p]) return;   // the same for every rank
  const ProbInfo pi = d.prob[p];
  const int nt = pi.nt, n = pi.n;
  const T* S = tptr<T>(d.S) + pi.s_off;
  T* b = tptr_mut<T>(d.b) + 6LL * pi.ext_begin;
  const T* Linv = tptr<T>(d.Linv) + (long long)p * d.max_nt * kTile * kTile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nown = nt > q ? (nt - q + R - 1) / R : 0;
  for (int e = tid; e < nown * kTile; e += blockDim.x) {
    const int lt = e / kTile, r = e % kTile, t = q + R * lt;
    ys[lt][r] = (kTile * t + r < n) ? b[kTile * t + r] : T(0);
  }
  // rows of step jj this warp handles first: i = q + R*warp
  T cur[kTile];
  auto fetch = [&](int jj) {
    const int i = q + R * warp;
    if (jj < 0 || i >= jj || warp >= 8) return;
    const int mj = tile_rows(n, jj);
    const T* row = S + (long long)kTile * jj * n + kTile * i + lane;
#pragma unroll
    for (int r = 0; r < kTile; ++r) cur[r] = r < mj ? row[(long long)r * n] : T(0);
  };
  // column `lane` of L_jj^-1 for the next diagonal tile this rank owns
  T lv[kTile];
  int jown = nt - 1 - ((nt - 1 - q) % R + R) % R;
  auto fetch_linv = [&](int jj) {
    if (jj < 0 || warp != kSolveOwnerWarp) return;
    const T* Lv = Linv + (long long)jj * kTile * kTile + lane;
#pragma unroll
    for (int r = 0; r < kTile; ++r) lv[r] = r >= lane ? Lv[r * kTile] : T(0);
  };
  fetch(nt - 1);
  fetch_linv(jown);
  if constexpr (R == 1) {
    __syncthreads();
  } else {   // every rank has started before its shared memory is written
    __syncthreads();
    cluster_arrive_relaxed();
    cluster_wait();
  }
  for (int j = nt - 1; j >= 0; --j) {
    const int par = j & 1;
    T s = T(0);
    const bool owner = (j == jown && warp == kSolveOwnerWarp);
    if (owner) {
      const T* y = ys[j / R];
#pragma unroll
      for (int r = 0; r < kTile; ++r) s += lv[r] * y[r];
      if constexpr (R == 1) {
        xb[par][lane] = s;
      } else {
        cg::cluster_group cluster = cg::this_cluster();
        for (int rk = 0; rk < R; ++rk) *cluster.map_shared_rank(&xb[par][lane], rk) = s;
        fence_cluster();
      }
    }
    if constexpr (R == 1) {
      __syncthreads();
    } else {
      cluster_arrive_relaxed();
      cluster_wait();
    }
    if (owner) {
      if (kTile * j + lane < n) b[kTile * j + lane] = s;
      jown -= R;
      fetch_linv(jown);
    }
    const int nact = warp < 8 && j > q ? (j - q + R - 1) / R : 0;   // (eight warps; others only keep step)
    if (warp < nact) {
      T acc = T(0);
#pragma unroll
      for (int r = 0; r < kTile; ++r) acc += cur[r] * xb[par][r];
      ys[warp][lane] -= acc;
    }
    for (int lt = warp + 8; lt < nact; lt += 8) {
      const int i = q + R * lt;
      const int mj = tile_rows(n, j);
      const T* row = S + (long long)kTile * j * n + kTile * i + lane;
      T acc = T(0);
      for (int r = 0; r < mj; ++r) acc += row[(long long)r * n] * xb[par][r];
      ys[lt][lane] -= acc;
    }
    fetch(j - 1);
    __syncthreads();
  }
}

// The cluster backward solve without a cluster-wide barrier per step.
// Rank q of the cluster owns the tile rows t = q (mod R) of y (local row
// lt = t / R) and warp w of the rank the local rows lt = w (mod 8).  Every
// rank keeps a slot per step j for delta_j and an mbarrier per step that
// completes once the 32 entries of delta_j have landed in the slot.  Step j
// (nt-1 down to 0): the warp owning row j forms delta_j = L_jj^-T y_j as
// soon as y_j is final (its last update, from step j+1, was this warp's
// own), and each of its lanes stores its entry into slot j of every rank
// with st.async, which counts the bytes against that rank's mbarrier j (no
// fence, no separate arrival).  Every warp waits on its own rank's
// mbarrier j (acquire), then subtracts L_ji^T delta_j from its rows i < j,
// the highest one (the next diagonal step's row when this warp owns it)
// from registers loaded one step ahead.  The per-row arithmetic is that of
// the single-CTA body.  Slots are not reused within a launch.  Waits are bounded
// (DevPlan::solve_spin_limit polls): a warp that gives up records a timeout
// in the problem's factor flag (the solve is void) and stops updating, but
// still sends its own deltas of the later steps; after a cluster barrier
// (every store issued) it waits, bounded again, for the stores into its rank
// that are still landing, so no CTA leaves while another writes into it.

template <typename T>
__host__ __device__ constexpr size_t solve_smem_bytes(int max_nt) {
  return size_t(max_nt) * 8 + size_t(max_nt) * kTile * sizeof(T) +
         size_t((max_nt + kSolveRanks - 1) / kSolveRanks) * kTile * sizeof(T);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
// An asynchronous store of v into rank `rank`'s copy of *dst that counts
// its bytes against that rank's copy of the mbarrier b (complete_tx): a
// waiter that sees the phase complete (acquire) sees the value.
template <typename T>
__device__ __forceinline__ void st_async_rank(T* dst, unsigned long long* b, int rank, T v) {
  unsigned ra, rb;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(smem_addr(dst)), "r"(rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(rb) : "r"(smem_addr(b)), "r"(rank));
  if constexpr (sizeof(T) == 4)
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n" ::"r"(ra),
                 "r"(__float_as_uint(v)), "r"(rb)
                 : "memory");
  else
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n" ::"r"(ra),
                 "l"(__double_as_longlong(v)), "r"(rb)
                 : "memory");
}
// This thread's arrival on b, announcing `bytes` of asynchronous stores.
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(b)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(unsigned long long* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void cluster_sync_acq_rel() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}

constexpr long long kSolveSpin = 1LL << 22;   // polls of a step's mbarrier (production)

// kProbe: the instantiation that reads the test controls of DevPlan
// (solve_spin_limit, solve_drop_step); production plans launch the other.
template <typename T, bool kProbe>
__global__ void __cluster_dims__(kSolveRanks, 1, 1) __launch_bounds__(256)
k_chol_solve(DevPlan d) {
  constexpr int R = kSolveRanks;
  const long long spin_limit = kProbe ? d.solve_spin_limit : kSolveSpin;
  const int drop_step = kProbe ? d.solve_drop_step : -1;
  extern __shared__ __align__(16) unsigned char solve_raw[];
  cg::cluster_group cluster = cg::this_cluster();
  const int q = int(cluster.block_rank());
  const int p = blockIdx.y;
  const LMState& st = d.state[p];
  if (!st.active || d.factor_flag[p]) return;   // the same for every rank
  const ProbInfo pi = d.prob[p];
  const int nt = pi.nt, n = pi.n, mt = d.max_nt;
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(solve_raw);   // [mt]
  T* xs = reinterpret_cast<T*>(bar + mt);                                         // [mt][kTile]
  T* ys = xs + size_t(mt) * kTile;                                                // [rows][kTile]
  const T* S = tptr<T>(d.S) + pi.s_off;
  T* b = tptr_mut<T>(d.b) + 6LL * pi.ext_begin;
  const T* Linv = tptr<T>(d.Linv) + (long long)p * d.max_nt * kTile * kTile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nown = nt > q ? (nt - q + R - 1) / R : 0;
  for (int e = tid; e < nown * kTile; e += blockDim.x) {
    const int lt = e / kTile, r = e % kTile, t = q + R * lt;
    ys[e] = (kTile * t + r < n) ? b[kTile * t + r] : T(0);
  }
  // barrier j completes when the owner's 32 stores of delta_j have landed
  for (int j = tid; j < nt; j += blockDim.x) {
    mbar_init(bar + j, 1);
    mbar_arrive_expect_tx(bar + j, unsigned(kTile * sizeof(T)));
  }
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  __syncthreads();
  cluster_sync_acq_rel();   // every rank's barriers exist before anyone arrives on them
  // the warp's rows, highest first: lt = lt_top, lt_top - 8, ...
  const int lt_top = warp < nown ? warp + 8 * ((nown - 1 - warp) / 8) : -1;
  // column `lane` of L_jj^-1 for the warp's next diagonal row
  T lv[kTile];
  auto fetch_linv = [&](int lt) {
    if (lt < 0) return;
    const T* Lv = Linv + (long long)(q + R * lt) * kTile * kTile + lane;
#pragma unroll
    for (int r = 0; r < kTile; ++r) lv[r] = r >= lane ? Lv[r * kTile] : T(0);
  };
  // L_ji (column `lane`) of the warp's highest row below j, loaded a step ahead
  T cur[kTile];
  int cur_lt = -1;
  auto fetch_cur = [&](int jj) {
    cur_lt = -1;
    if (jj < 0 || lt_top < 0) return;
    int lt = lt_top;
    while (lt >= 0 && q + R * lt >= jj) lt -= 8;
    if (lt < 0) return;
    cur_lt = lt;
    const int mj = tile_rows(n, jj);
    const T* row = S + (long long)kTile * jj * n + kTile * (q + R * lt) + lane;
#pragma unroll
    for (int r = 0; r < kTile; ++r) cur[r] = r < mj ? row[(long long)r * n] : T(0);
  };
  fetch_linv(lt_top);
  fetch_cur(nt - 1);
  int next_diag = lt_top;   // the warp's next diagonal row (local index)
  int j_fail = -1;
  for (int j = nt - 1; j >= 0; --j) {
    if (next_diag >= 0 && q + R * next_diag == j) {
      __syncwarp();   // y_j's entries are this warp's own, written in step j+1
      const T* y = ys + next_diag * kTile;
      T sj = T(0);
#pragma unroll
      for (int r = 0; r < kTile; ++r) sj += lv[r] * y[r];
      if (j != drop_step)
        for (int rk = 0; rk < R; ++rk) st_async_rank(xs + (size_t)j * kTile + lane, bar + j, rk, sj);
      if (kTile * j + lane < n) b[kTile * j + lane] = sj;
      next_diag -= 8;
      fetch_linv(next_diag);
    }
    long long spin = 0;
    while (!mbar_try_wait_cluster(bar + j, 0u))
      if (++spin > spin_limit) break;
    if (spin > spin_limit) {   // delta_j did not come: the solve is void
      if (lane == 0) d.factor_flag[p] = 2;
      j_fail = j;
      break;
    }
    const T* xj = xs + (size_t)j * kTile;
    if (cur_lt >= 0) {
      T acc = T(0);
#pragma unroll
      for (int r = 0; r < kTile; ++r) acc += cur[r] * xj[r];
      ys[cur_lt * kTile + lane] -= acc;
      for (int lt = cur_lt - 8; lt >= 0; lt -= 8) {   // the warp's other rows below j
        const int mj = tile_rows(n, j);
        const T* row = S + (long long)kTile * j * n + kTile * (q + R * lt) + lane;
        T a2 = T(0);
        for (int r = 0; r < mj; ++r) a2 += row[(long long)r * n] * xj[r];
        ys[lt * kTile + lane] -= a2;
      }
    }
    fetch_cur(j - 1);
  }
  if (j_fail >= 0) {
    // the warp gave up at step j_fail: it still sends its own deltas of the
    // steps below (void values), so every delta another warp waits for is sent
    for (int j = j_fail - 1; j >= 0; --j) {
      if (next_diag >= 0 && q + R * next_diag == j) {
        if (j != drop_step)
          for (int rk = 0; rk < R; ++rk) st_async_rank(xs + (size_t)j * kTile + lane, bar + j, rk, T(0));
        next_diag -= 8;
      }
    }
  }
  __syncthreads();
  cluster_sync_acq_rel();   // every rank has issued all of its stores
  if (j_fail >= 0) {
    // wait (bounded) for the stores into this rank that are still landing
    // before the CTA may leave
    for (int j = 0; j < nt; ++j) {
      long long spin = 0;
      while (!mbar_try_wait_cluster(bar + j, 0u) && ++spin <= spin_limit) {
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_chol_solve_small(DevPlan d) {
  chol_solve_body<T, 1>(d, 0);
}

// Factorization and solve of small reduced systems (at most
// kSolveSmallTiles tile rows, FP32), batched or alone: one CTA of 16 warps per
// problem keeps the tiles of the lower triangle in shared memory and runs the
// schedule of the per-column launches (k_chol_step) inside the CTA.  For each
// column c: the panels L_ic = A_ic L_cc^-T, a tile to a group of four warps;
// then group 0 updates the next diagonal tile and factors it while the other
// groups take the rest of the trailing updates A_ij -= L_ic L_jc^T, the
// panels into S and the forward-solve updates b_i -= L_ic y_c.  The
// per-element arithmetic is that of k_chol_step, so the bits are those of
// k_chol_step and k_chol_dataflow; then the backward solve of
// k_chol_solve_small.  With two groups, one after the other through every
// phase, 512 windows took 192 us an iteration instead of 148.
constexpr int kCholSmallThreads = 512;

template <typename T>
__host__ __device__ constexpr size_t chol_small_smem(int max_nt) {
  return size_t(max_nt) * (max_nt + 1) / 2 * sizeof(Tile<T>);
}

template <typename T>
__global__ void __launch_bounds__(kCholSmallThreads, 1) k_chol_small(DevPlan d) {
  constexpr int kGroups = kCholSmallThreads / 128;
  extern __shared__ __align__(16) unsigned char cs_raw[];
  __shared__ __align__(16) Tile<T> Dinv[2];
  __shared__ T bs[kSolveSmallTiles][kTile];   // b after the columns done so far
  __shared__ PotrfBuf<T> fb;
  __shared__ int ok_s;
  Tile<T>* A = reinterpret_cast<Tile<T>*>(cs_raw);   // tile (i, j), j <= i, at i (i + 1) / 2 + j
  const int p = blockIdx.y;
  const LMState& st = d.state[p];
  if (!st.active || d.factor_flag[p]) return;
  const ProbInfo pi = d.prob[p];
  const int nt = pi.nt, n = pi.n;
  if (nt > kSolveSmallTiles || nt > d.max_nt) {   // (never: the planner's bound) fail loudly
    if (threadIdx.x == 0) d.factor_flag[p] = 1;
    return;
  }
  T* S = tptr_mut<T>(d.S) + pi.s_off;
  T* b = tptr_mut<T>(d.b) + 6LL * pi.ext_begin;
  T* Lg = tptr_mut<T>(d.Linv) + (long long)p * d.max_nt * kTile * kTile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = tid >> 7, gt = tid & 127, gw = warp & 3;
  auto at = [&](int i, int j) -> Tile<T>& { return A[i * (i + 1) / 2 + j]; };
  auto row_of = [](int lin) {   // the row of tile `lin` of a lower triangle
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= lin) ++i;
    return i;
  };
  // the tiles, two per group in flight; a diagonal tile keeps its lower
  // triangle and has identity rows past the matrix
  const int ntiles = nt * (nt + 1) / 2;
  for (int lin0 = g; lin0 < ntiles; lin0 += 2 * kGroups) {
    T v[2][8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int lin = lin0 + h * kGroups;
      if (lin >= ntiles) continue;
      const int i = row_of(lin), j = lin - i * (i + 1) / 2, mi = tile_rows(n, i);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int r = gw + 4 * u;
        const bool in = r < mi && (i != j || lane <= r);
        v[h][u] = in ? S[(long long)(kTile * i + r) * n + kTile * j + lane]
                     : (i == j && r >= mi && r == lane ? T(1) : T(0));
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int lin = lin0 + h * kGroups;
      if (lin >= ntiles) continue;
#pragma unroll
      for (int u = 0; u < 8; ++u) A[lin][gw + 4 * u][lane] = v[h][u];
    }
  }
  if (tid == 0) {
    ok_s = 1;
    fb.step = 0;
  }
  for (int e = tid; e < nt * kTile; e += blockDim.x) {
    const int t = e / kTile, r = e % kTile;
    bs[t][r] = r < tile_rows(n, t) ? b[kTile * t + r] : T(0);
  }
  __syncthreads();
  auto factor = [&](int c) {   // group 0
    if (!tile_potrf_inverse(at(c, c), Dinv[c & 1], fb, Lg + (long long)c * kTile * kTile, gw, lane) && lane == 0)
      ok_s = 0;
  };
  for (int c = -1; c < nt; ++c) {
    if (c >= 0) {
      // panels, a tile to a group; y_c = L_cc^-1 b_c (b_c after the columns before c)
      const Tile<T>& Li = Dinv[c & 1];
      for (int i = c + 1 + g; i < nt; i += kGroups) {
        T sv[kTile / 4];
        tile_panel_sums<T, 4>(at(i, c), Li, gw, lane, sv);
        bar_sync(kQuadBarrier + g, 128);   // every read of this tile precedes its writes
#pragma unroll
        for (int u = 0; u < kTile / 4; ++u) at(i, c)[lane][panel_col<4>(u, gw)] = sv[u];
      }
      if (warp == 15) {
        T y = T(0);
#pragma unroll 8
        for (int q = 0; q < kTile; ++q) y += Li[lane][q] * bs[c][q];
        __syncwarp();
        bs[c][lane] = y;
        if (lane < tile_rows(n, c)) b[kTile * c + lane] = y;
      }
      __syncthreads();
    }
    if (c + 1 < nt) {
      if (g == 0) {
        if (c >= 0) {
          tile_sub_sym(at(c + 1, c + 1), at(c + 1, c));
          bar_sync(kQuadBarrier, 128);
        }
        factor(c + 1);
      } else if (c >= 0) {
        // the other trailing tiles (lin 0 is the next diagonal one)
        const int m = nt - c - 1, ntr = m * (m + 1) / 2;
        for (int lin = g; lin < ntr; lin += kGroups - 1) {
          const int ti = row_of(lin), i = c + 1 + ti, j = c + 1 + (lin - ti * (ti + 1) / 2);
          tile_sub_xyt_t<T>(at(i, j), at(i, c), at(j, c), gt);
        }
        // the panels into S for the backward solve, b_i -= L_ic y_c below
        for (int i = c + g; i < nt; i += kGroups - 1) {
          const int mi = tile_rows(n, i);
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int r = gw + 4 * u;
            if (r < mi) S[(long long)(kTile * i + r) * n + kTile * c + lane] = at(i, c)[r][lane];
          }
          if (gw == 3) {
            T t = bs[i][lane];
#pragma unroll 8
            for (int q = 0; q < kTile; ++q) t -= at(i, c)[lane][q] * bs[c][q];
            bs[i][lane] = t;
          }
        }
      }
    }
    __syncthreads();
    if (!ok_s) {
      if (tid == 0) d.factor_flag[p] = 1;
      return;
    }
  }
  chol_solve_body<T, 1>(d, 0);
}

// ---------------------------------------------------------------------------
// Block-Jacobi PCG on the block-sparse reduced system (large scenes).  The
// reduced system keeps one 6x6 block per co-visible image pair (first image
// <= second): Sblk[blk][6x + y] is the row of component x of the first image
// and the column of component y of the second.  The matrix-vector product
// runs one warp per image over the blocks touching it (each block read from
// both ends, no atomics); all sums have a fixed order, so a problem's
// iterates are the same alone and in a batch.  The solution overwrites b.
// Per problem and iteration: p.q, r.z, r.r and b.b are reduced from per-chunk
// partials (chunks of kImageChunk images) by every CTA that needs them.
// ---------------------------------------------------------------------------
// Slots slot[0 .. N) of problem p's chunk partials, each summed over its chunks
// (thread t takes chunks t, t + 256, ..., then the tree of block_sum), into
// out[0 .. N) in every thread: one pass and two barriers for all of them (an
// FP64 addition takes 64 cycles, and every CTA waits for these sums before
// its own work).  red [9 N].
template <int N>
__device__ __forceinline__ void pcg_prob_sums(const DevPlan& d, int p, const int (&slot)[N], double* red,
                                              double (&out)[N]) {
  double v[N];
#pragma unroll
  for (int e = 0; e < N; ++e) v[e] = 0.0;
  for (int c = d.prob_ext_chunk_off[p] + threadIdx.x; c < d.prob_ext_chunk_off[p + 1]; c += blockDim.x) {
    const double* part = d.pcg_part + (long long)kPcgSlots * c;
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] += part[slot[e]];
  }
  const double tot = block_sums<N>(v, red);
  if (threadIdx.x < N) red[8 * N + threadIdx.x] = tot;
  __syncthreads();
#pragma unroll
  for (int e = 0; e < N; ++e) out[e] = red[8 * N + e];
}

// Six consecutive values (three 8-byte or 16-byte loads).
template <typename T>
__device__ __forceinline__ void load6(const T* __restrict__ p, T* o) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const auto v = reinterpret_cast<const typename Pair2<T>::type*>(p)[c];
    o[2 * c] = v.x;
    o[2 * c + 1] = v.y;
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_assemble_blocks(DevPlan d) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= 36LL * d.n_blocks) return;
  const int blk = int(e / 36), el = int(e % 36);
  const int2 g = __ldg(d.blk_gij + blk);   // global reduced-system images, g.x <= g.y
  const int p = __ldg(d.ext_prob + g.x);
  const LMState& st = d.state[p];
  if (!st.active) return;
  const ProbInfo& pi = d.prob[p];
  const int ib = __ldg(d.blk_item_off + blk), ie = __ldg(d.blk_item_off + blk + 1);
  double v = 0.0;
  for (int t = ib; t < ie; ++t) v += d.item_partial[(long long)kItemStride * t + el];
  double sv = -v;
  // entry (component el / 6 of g.x, component el % 6 of g.y); the base of
  // the symmetric system is read as row (g.y, el % 6), column (g.x, el / 6)
  const int lx = g.x - pi.ext_begin, ly = g.y - pi.ext_begin;
  if (ly < pi.num_images) {
    if (g.x == g.y) sv += d.U[36LL * (pi.image_begin + lx) + el];
  } else {
    sv += reduced_base(d, pi, ly, el % 6, lx, el / 6);
  }
  if (g.x == g.y && el % 7 == 0) sv += st.mu;
  tptr_mut<T>(d.Sblk)[36LL * blk + el] = T(sv);
  if (g.x == g.y && el < 6) {
    double rv = 0.0;
    for (int t = ib; t < ie; ++t) rv += d.item_partial[(long long)kItemStride * t + 36 + el];
    tptr_mut<T>(d.b)[6LL * g.x + el] = T(reduced_grad(d, pi, lx, el) - rv);
  }
}

// Inverse of each image's diagonal block (6x6 Cholesky, then L^-T L^-1).
template <typename T>
__global__ void __launch_bounds__(128) k_pcg_precond(DevPlan d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.I_ext) return;
  const int p = d.ext_prob[i];
  if (!d.state[p].active) return;
  const T* A = tptr<T>(d.Sblk) + 36LL * d.img_diag_blk[i];
  T L[6][6], X[6][6];
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    T sjj = A[7 * j];
#pragma unroll
    for (int k = 0; k < j; ++k) sjj -= L[j][k] * L[j][k];
    ok = ok && sjj > T(0);
    const T ljj = sqrt(sjj > T(0) ? sjj : T(1));
    const T rj = T(1) / ljj;
    L[j][j] = ljj;
#pragma unroll
    for (int r = j + 1; r < 6; ++r) {
      T sr = A[6 * r + j];
#pragma unroll
      for (int k = 0; k < j; ++k) sr -= L[r][k] * L[j][k];
      L[r][j] = sr * rj;
    }
  }
  // X = L^-1 (lower), column by column
#pragma unroll
  for (int c = 0; c < 6; ++c) {
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      if (r < c) {
        X[r][c] = T(0);
        continue;
      }
      T v = (r == c) ? T(1) : T(0);
#pragma unroll
      for (int k = c; k < r; ++k) v -= L[r][k] * X[k][c];
      X[r][c] = v / L[r][r];
    }
  }
  T* M = tptr_mut<T>(d.Minv) + 36LL * i;
#pragma unroll
  for (int x = 0; x < 6; ++x)
#pragma unroll
    for (int y = 0; y < 6; ++y) {
      T v = T(0);
#pragma unroll
      for (int k = 0; k < 6; ++k) v += X[k][x] * X[k][y];
      M[6 * x + y] = v;
    }
  if (!ok) atomicExch(d.factor_flag + p, 1);
}

// z = Minv r for this warp's image: lanes 0..5 hold r and return z.
template <typename T>
__device__ __forceinline__ T pcg_precond_apply(const DevPlan& d, int img, T rv, int lane) {
  const T* M = tptr<T>(d.Minv) + 36LL * img;
  T z = T(0);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const T rk = __shfl_sync(0xffffffffu, rv, k);
    if (lane < 6) z += M[6 * lane + k] * rk;
  }
  return z;
}

// x = 0 (in b), r = b, z = Minv r, p_0 = 0; partials r.z, r.r, b.b.
template <typename T>
__global__ void __launch_bounds__(256) k_pcg_init(DevPlan d) {
  __shared__ double red[33];
  if (d.pcg_it && blockIdx.x == 0 && threadIdx.x == 0) *d.pcg_it = 0;   // the device-side loop's count
  const Chunk ch = d.ext_chunks[blockIdx.x];
  const LMState& st = d.state[ch.prob];
  if (!st.active || d.factor_flag[ch.prob]) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int img = ch.begin + warp;
  double rz = 0.0, rr = 0.0;
  if (img < ch.end) {
    T* b = tptr_mut<T>(d.b);
    const T rv = lane < 6 ? b[6LL * img + lane] : T(0);
    const T z = pcg_precond_apply<T>(d, img, rv, lane);
    if (lane < 6) {
      b[6LL * img + lane] = T(0);
      tptr_mut<T>(d.pcg_r)[6LL * img + lane] = rv;
      tptr_mut<T>(d.pcg_z)[6LL * img + lane] = z;
      tptr_mut<T>(d.pcg_p[0])[6LL * img + lane] = T(0);
      rz = double(rv) * double(z);
      rr = double(rv) * double(rv);
    }
  }
  double sums[2] = {rz, rr};
  const double tot = block_sums<2>(sums, red);
  double* part = d.pcg_part + (long long)kPcgSlots * blockIdx.x;
  if (threadIdx.x == 0) {
    part[1] = tot;
    part[6] = 0.0;
    if (blockIdx.x == d.prob_ext_chunk_off[ch.prob]) d.pcg_done[ch.prob] = 0;
  } else if (threadIdx.x == 1) {
    part[3] = tot;
    part[5] = tot;
  }
}

// Iteration it, part 1: beta from the last two r.z, p = z + beta p_old (own
// images stored, neighbours' formed on the fly), q = S p, partial p.q.
template <typename T>
__global__ void __launch_bounds__(256) k_pcg_spmv(DevPlan d, int it, int loop) {
  __shared__ double red[9 * 4];
  // in the device-side loop `it` is the half (0, 1) of the loop body's pass
  if (loop) it += 2 * *reinterpret_cast<volatile int*>(d.pcg_it);
  if (it >= d.pcg_max_iterations) return;
  const Chunk ch = d.ext_chunks[blockIdx.x];
  const int p = ch.prob;
  const LMState& st = d.state[p];
  if (!st.active || d.factor_flag[p] || d.pcg_done[p]) return;
  const int par = it & 1;
  // r.z, r.r, b.b and (from the second iteration on) the last r.z
  const int slot[4] = {1 + par, 3 + par, 5, it > 0 ? 1 + (par ^ 1) : 5};
  double sum[4];
  pcg_prob_sums<4>(d, p, slot, red, sum);
  if (sum[1] <= d.pcg_tol2 * sum[2]) return;          // converged (or b = 0)
  const T beta = it > 0 ? T(sum[0] / sum[3]) : T(0);
  const T* z = tptr<T>(d.pcg_z);
  const T* pold = tptr<T>(d.pcg_p[par]);
  T* pnew = tptr_mut<T>(d.pcg_p[par ^ 1]);
  const T* Sb = tptr<T>(d.Sblk);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int img = ch.begin + warp;
  double dot = 0.0;
  if (img < ch.end) {
    T acc[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
    const int a0 = __ldg(d.adj_off + img), a1 = __ldg(d.adj_off + img + 1);
    for (int e = a0 + lane; e < a1; e += 32) {
      const int2 en = __ldg(d.adj + e);
      const int j = en.y >> 1;
      // (the block in 16-byte loads: entry by entry, a warp's 36 loads of
      // scattered 144-byte blocks took three quarters of the kernel)
      T pj[6], po[6], B[36];
      load6(z + 6LL * j, pj);
      load6(pold + 6LL * j, po);
      load_vec<36>(Sb + 36LL * en.x, B);
#pragma unroll
      for (int c = 0; c < 6; ++c) pj[c] = pj[c] + beta * po[c];
      if (!(en.y & 1)) {
#pragma unroll
        for (int x = 0; x < 6; ++x)
#pragma unroll
          for (int y = 0; y < 6; ++y) acc[x] += B[6 * x + y] * pj[y];
      } else {
#pragma unroll
        for (int x = 0; x < 6; ++x)
#pragma unroll
          for (int y = 0; y < 6; ++y) acc[y] += B[6 * x + y] * pj[x];
      }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = warp_sum_t<T>(acc[c]);
    if (lane < 6) {
      T qv = acc[0];
#pragma unroll
      for (int c = 1; c < 6; ++c)
        if (lane == c) qv = acc[c];
      const T pv = z[6LL * img + lane] + beta * pold[6LL * img + lane];
      pnew[6LL * img + lane] = pv;
      tptr_mut<T>(d.pcg_q)[6LL * img + lane] = qv;
      dot = double(pv) * double(qv);
    }
  }
  __syncthreads();   // (red is read above)
  double sums[1] = {dot};
  dot = block_sums<1>(sums, red);
  if (threadIdx.x == 0) d.pcg_part[(long long)kPcgSlots * blockIdx.x] = dot;
}

// Iteration it, part 2: alpha = r.z / p.q, x += alpha p, r -= alpha q,
// z = Minv r, partials of the next r.z and r.r.
template <typename T>
__global__ void __launch_bounds__(256) k_pcg_update(DevPlan d, int it, int loop) {
  __shared__ double red[9 * 4];
  if (loop) it += 2 * *reinterpret_cast<volatile int*>(d.pcg_it);
  if (it >= d.pcg_max_iterations) return;
  const Chunk ch = d.ext_chunks[blockIdx.x];
  const int p = ch.prob;
  LMState& st = d.state[p];
  if (!st.active || d.factor_flag[p] || d.pcg_done[p]) return;
  const bool lead = blockIdx.x == d.prob_ext_chunk_off[p];
  const int par = it & 1;
  // r.z, r.r, b.b, p.q (the last one stale, and not looked at, once converged)
  const int slot[4] = {1 + par, 3 + par, 5, 0};
  double sum[4];
  pcg_prob_sums<4>(d, p, slot, red, sum);
  const double rz = sum[0], rr = sum[1], bb = sum[2], pq = sum[3];
  double* part = d.pcg_part + (long long)kPcgSlots * blockIdx.x;
  if (rr <= d.pcg_tol2 * bb) {
    // converged: carry this chunk's partials to the next parity so that
    // every later iteration sees the same sums and returns as well
    if (threadIdx.x == 0) {
      part[1 + (par ^ 1)] = part[1 + par];
      part[3 + (par ^ 1)] = part[3 + par];
      if (lead) d.pcg_done[p] = 1;   // later launches return at once
    }
    return;
  }
  if (!(pq > 0.0)) {
    // breakdown (the residual is at the rounding floor): keep x and stop, by
    // zeroing the next r.r, which the branch above then carries forward
    if (threadIdx.x == 0) {
      part[1 + (par ^ 1)] = part[1 + par];
      part[3 + (par ^ 1)] = 0.0;
    }
    return;
  }
  const T alpha = T(rz / pq);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int img = ch.begin + warp;
  double rzn = 0.0, rrn = 0.0, xr = 0.0;
  if (img < ch.end) {
    const long long o = 6LL * img + (lane < 6 ? lane : 0);
    T rv = T(0);
    if (lane < 6) {
      T* x = tptr_mut<T>(d.b);
      T* r = tptr_mut<T>(d.pcg_r);
      const T pv = tptr<T>(d.pcg_p[par ^ 1])[o];
      const T qv = tptr<T>(d.pcg_q)[o];
      const T xv = x[o] + alpha * pv;
      x[o] = xv;
      rv = r[o] - alpha * qv;
      r[o] = rv;
      xr = double(xv) * double(rv);
    }
    const T z = pcg_precond_apply<T>(d, img, rv, lane);
    if (lane < 6) {
      tptr_mut<T>(d.pcg_z)[o] = z;
      rzn = double(rv) * double(z);
      rrn = double(rv) * double(rv);
    }
  }
  __syncthreads();   // (red is read above)
  double sums[3] = {rzn, rrn, xr};
  const double tot = block_sums<3>(sums, red);
  if (threadIdx.x == 0) {
    part[1 + (par ^ 1)] = tot;
    if (lead) st.pcg_iters += 1;
  } else if (threadIdx.x == 1) {
    part[3 + (par ^ 1)] = tot;
  } else if (threadIdx.x == 2) {
    part[6] = tot;
  }
}

// The device-side PCG loop (a CUDA-graph while node): after each pass of
// two iterations one warp counts the pass and ends the loop once every
// problem's inner solve has stopped (converged, broken down, not solving)
// or the iterations are used up.
__global__ void __launch_bounds__(32) k_pcg_loop_ctrl(DevPlan d, cudaGraphConditionalHandle h) {
  const int m = *reinterpret_cast<volatile int*>(d.pcg_it) + 1;
  bool more = 2 * m < d.pcg_max_iterations;
  if (more) {
    bool open = false;
    for (int p = threadIdx.x; p < d.B && !open; p += 32) {
      const LMState& st = d.state[p];
      open = st.active && !d.factor_flag[p] && !d.pcg_done[p];
    }
    more = __any_sync(0xffffffffu, open);
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    *d.pcg_it = m;
    if (more) ++*d.pcg_extra;
    cudaGraphSetConditional(h, more ? 1u : 0u);
  }
}

// A loop inside another loop's body: a node's condition takes its default
// only when the whole graph is launched, so it is opened before each solve.
__global__ void k_pcg_loop_open(cudaGraphConditionalHandle h) { cudaGraphSetConditional(h, 1u); }

// ---------------------------------------------------------------------------
// back-substitution and update
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kPointChunk, sizeof(T) == sizeof(float) ? 10 : 0) k_backsub(DevPlan d) {
  __shared__ double red[32];
  __shared__ T prod[3][kPointKeys];   // J_p^T (J_i delta_i) of the chunk's keys
  // With DevPlan::fold_ctrl the last CTA of a problem to finish runs the LM
  // step decision (k_ctrl_step's body), so every CTA of an active problem
  // arrives, also when the factorization failed and there is nothing to do.
  const int prob = blockIdx.x < d.n_pt_chunks ? d.pt_chunks[blockIdx.x].prob
                                              : d.img_chunks[blockIdx.x - d.n_pt_chunks].prob;
  if (!d.state[prob].active) return;
  const bool failed = d.factor_flag[prob] != 0;
  if (failed) {
    // nothing to compute
  } else if (blockIdx.x < d.n_pt_chunks) {
    const Chunk ch = d.pt_chunks[blockIdx.x];
    const LMState& st = d.state[ch.prob];
    const int par = st.parity;
    const int pt = ch.begin + threadIdx.x;
    double dn2 = 0.0, xn2 = 0.0, gd = 0.0;
    // w = sum over the point's keys of J_p^T (J_i delta_i) from the Jacobian
    // records, then t = C^-1 (g - w) with C^-1 g = h.  The products are formed
    // a key to a thread (the chunk's records are consecutive, every lane has a
    // key, no load waits for another key's) and added point by point, in key
    // order, from shared memory.  A point to a thread throughout, a warp
    // walked its longest track, two dependent loads a key: 512 windows 764 us
    // instead of 647, random walk 349 instead of 239.  The loads' latency
    // bounds it (DRAM 48% busy at 29 warps an SM), so FP32 is held to 48
    // registers for 40 warps: 586 and 228 us.
    T w0 = T(0), w1 = T(0), w2 = T(0);
    {
      const T* __restrict__ JR = tptr<T>(d.JR[par]);
      const T* __restrict__ delta = tptr<T>(d.b);
      const int k0 = __ldg(d.pt_key_off + ch.begin), k1 = __ldg(d.pt_key_off + ch.end);
      const int kb = pt < ch.end ? __ldg(d.pt_key_off + pt) : k1, ke = pt < ch.end ? __ldg(d.pt_key_off + pt + 1) : k1;
      for (int base = k0; base < k1; base += kPointKeys) {
        const int top = min(k1, base + kPointKeys);
        for (int k = base + int(threadIdx.x); k < top; k += kPointChunk) {
          T rec[kJRStride], dl[6];
          load_vec<kJRStride>(JR + (long long)kJRStride * k, rec);
          const int ext = d.img_ext ? __ldg(d.img_ext + __ldg(d.key_img + k)) : __ldg(d.key_img + k);
          load6(delta + 6LL * ext, dl);
          T u0 = T(0), u1 = T(0);
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            u0 += rec[6 + c] * dl[c];
            u1 += rec[12 + c] * dl[c];
          }
          prod[0][k - base] = rec[0] * u0 + rec[3] * u1;
          prod[1][k - base] = rec[1] * u0 + rec[4] * u1;
          prod[2][k - base] = rec[2] * u0 + rec[5] * u1;
        }
        __syncthreads();
        const int e1 = min(ke, top) - base;
        for (int e = max(kb, base) - base; e < e1; ++e) {
          w0 += prod[0][e];
          w1 += prod[1][e];
          w2 += prod[2][e];
        }
        if (top < k1) __syncthreads();   // (before the next part overwrites them)
      }
    }
    if (pt < ch.end) {
      T ps[12];
      load_vec<12>(tptr<T>(d.PS) + 12LL * pt, ps);
      const T i00 = ps[0], m10 = ps[1], i11 = ps[2], m20 = ps[3], m21 = ps[4], i22 = ps[5];
      T t0 = ps[6] - i00 * w0, t1 = ps[7] - (m10 * w0 + i11 * w1), t2 = ps[8] - (m20 * w0 + m21 * w1 + i22 * w2);
      // free cameras: the point's camera records (Z = C^-1 W) against their
      // reduced-system images' deltas
      if (d.pt_rec_off) {
        const T* __restrict__ Z = tptr<T>(d.Z);
        const int rb = __ldg(d.pt_rec_off + pt), re = __ldg(d.pt_rec_off + pt + 1);
        for (int r = rb; r < re; ++r) {
          T z[kZStride];
          load_z(d, Z, r, z);
          const T* di = tptr<T>(d.b) + 6LL * __ldg(&d.rec_info[r - d.K].y);
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            const T dl = di[c];
            t0 -= z[c] * dl;
            t1 -= z[6 + c] * dl;
            t2 -= z[12 + c] * dl;
          }
        }
      }
      // delta = C^-T t, C^-1 rows [i00 0 0; m10 i11 0; m20 m21 i22]
      const double dp[3] = {double(i00 * t0 + m10 * t1 + m20 * t2), double(i11 * t1 + m21 * t2),
                            double(i22 * t2)};
      T pv[12];
      load_vec<12>(tptr<T>(d.PV) + 12LL * pt, pv);
      const double* x = d.x_pt[par] + 3LL * pt;
      double* xn = d.x_pt[1 - par] + 3LL * pt;
      float2* xf = d.x_ff[1 - par] ? d.x_ff[1 - par] + 3LL * pt : nullptr;
      const bool free_pt = !(d.prob[ch.prob].fix & 1);   // a fixed point is not in x
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        xn[a] = x[a] - dp[a];
        if (xf) xf[a] = ff_split(xn[a]);
        dn2 += dp[a] * dp[a];
        if (free_pt) xn2 += x[a] * x[a];
        gd += double(pv[6 + a]) * dp[a];
      }
    }
    double sums[3] = {dn2, xn2, gd};
    const double tot = block_sums<3>(sums, red);
    if (threadIdx.x < 3) d.pt_chunk_sum[3LL * blockIdx.x + threadIdx.x] = tot;
  } else {
    const int c = blockIdx.x - d.n_pt_chunks;
    const Chunk ch = d.img_chunks[c];
    const LMState& st = d.state[ch.prob];
    const int par = st.parity;
    double dn2 = 0.0, xn2 = 0.0, gd = 0.0;
    const long long e0 = 6LL * ch.begin, e1 = 6LL * ch.end;
    const ProbInfo& pi = d.prob[ch.prob];
    const long long boff = 6LL * (pi.ext_begin - pi.image_begin);
    const bool free_img = !(pi.fix & 2);   // fixed images are not in x
    for (long long e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
      double dv = double(tptr<T>(d.b)[e + boff]), xv = d.x_img[par][e];
      d.x_img[1 - par][e] = xv - dv;
      dn2 += dv * dv;
      if (free_img) xn2 += xv * xv;
      gd += d.gi[e] * dv;
    }
    double sums[3] = {dn2, xn2, gd};
    const double tot = block_sums<3>(sums, red);
    // the candidate's rotations (the barrier made x_img[1 - par] visible)
    if (threadIdx.x < ch.end - ch.begin) image_prep_one<T>(d, ch.begin + threadIdx.x, 1 - par);
    if (threadIdx.x < 3) d.img_chunk_sum[3LL * c + threadIdx.x] = tot;
  }
  if (d.fold_ctrl) {
    __shared__ int last;
    const int total = d.prob_pt_chunk_off[prob + 1] - d.prob_pt_chunk_off[prob] +
                      d.prob_img_chunk_off[prob + 1] - d.prob_img_chunk_off[prob];
    if (last_arrival(d.fold_count + 2 * prob, total, &last)) ctrl_step_body<true>(d, prob, red);
  }
}

// Free cameras: delta_c from the camera's parts of the reduced-system
// solution, the candidate x_c - delta_c, and the camera's terms of
// ||delta||^2, ||x||^2 and g^T delta.
template <typename T>
__global__ void k_cam_backsub(DevPlan d) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d.Ctot) return;
  const int4 ci = d.cam_info[c];
  const LMState& st = d.state[ci.z];
  if (!st.active || d.factor_flag[ci.z]) return;
  double dn2 = 0.0, xn2 = 0.0, gd = 0.0;
  if (ci.x > 0) {
    const int par = st.parity;
    const T* b = tptr<T>(d.b) + 6LL * ci.w;
    for (int m = 0; m < ci.x; ++m) {
      const double dv = double(b[m]), xv = d.x_cam[par][10LL * c + m];
      d.x_cam[1 - par][10LL * c + m] = xv - dv;
      dn2 += dv * dv;
      xn2 += xv * xv;
      gd += d.gc[10LL * c + m] * dv;
    }
  }
  d.cam_sum[3LL * c] = dn2;
  d.cam_sum[3LL * c + 1] = xn2;
  d.cam_sum[3LL * c + 2] = gd;
}

// ---------------------------------------------------------------------------
// LM control (one warp per problem)
// ---------------------------------------------------------------------------
// Sum of one field of a problem's chunk partials by the whole CTA (thread t
// adds chunks t, t + blockDim, ... in order, then a fixed-shape tree):
// deterministic, and each thread waits on a few loads instead of one warp
// walking hundreds of chunks.  Result valid in thread 0.
// CG: the partials were written by other CTAs of the running kernel, so
// they are read through L2 (ld.global.cg), never from a stale L1 line.
template <bool CG = false>
__device__ double prob_sum(const double* v, int stride, int off, const int* chunk_off, int p,
                           double* red) {
  double s = 0.0;
  for (int c = chunk_off[p] + threadIdx.x; c < chunk_off[p + 1]; c += blockDim.x)
    s += CG ? __ldcg(v + (long long)stride * c + off) : v[(long long)stride * c + off];
  return block_sum(s, red);
}

// The first NF fields of a problem's chunk partials (stride fields per
// chunk) summed in one pass: each thread walks its chunks with NF loads per
// chunk, four chunks in flight, then fixed-shape trees.  Results in thread 0.
template <int NF, bool CG = false>
__device__ void prob_sums(const double* v, int stride, const int* chunk_off, int p, double* red,
                          double* out) {
  double s[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) s[f] = 0.0;
  const int c0 = chunk_off[p], c1 = chunk_off[p + 1];
#pragma unroll 4
  for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
#pragma unroll
    for (int f = 0; f < NF; ++f)
      s[f] += CG ? __ldcg(v + (long long)stride * c + f) : v[(long long)stride * c + f];
  }
#pragma unroll
  for (int f = 0; f < NF; ++f) out[f] = block_sum(s[f], red);
}

// LM control: one CTA per problem (kCtrlThreads), thread 0 decides.
constexpr int kCtrlThreads = 256;

__global__ void __launch_bounds__(kCtrlThreads) k_ctrl_initial_cost(DevPlan d) {
  __shared__ double red[32];
  const int p = blockIdx.x;
  LMState& st = d.state[p];
  if (!st.active) return;
  double fr[2];
  prob_sums<2>(d.key_chunk_sum, 2, d.prob_key_chunk_off, p, red, fr);
  if (threadIdx.x != 0) return;
  double F = fr[0];
  const double raw = fr[1];
  if (d.cons_cost) F += d.cons_cost[p];
  st.F = F;
  st.raw = raw;
  st.initial_cost = F;
  if (!isfinite(F)) {
    st.status = GBA_ERR_NAN;
    st.stop = GBA_STOP_ERROR;
    st.active = 0;
  }
}

// The checks after problem p's linearization; whether it goes on.
__device__ __forceinline__ bool ctrl_after_linearize(const DevPlan& d, int p) {
  LMState& st = d.state[p];
  if (st.relin && st.active) {
    const double ginf = bitsd(st.ginf_bits);
    if (st.first) {
      st.mu = d.tau * bitsd(st.maxdiag_bits);
      st.first = 0;
    }
    if (ginf <= d.eps1) {
      st.active = 0;
      st.stop = GBA_STOP_SMALL_GRADIENT;
    }
  }
  st.relin = 0;
  if (st.active && st.iter >= d.max_iterations) {
    st.active = 0;
    st.stop = GBA_STOP_MAX_ITERATIONS;
  }
  return st.active != 0;
}

__global__ void k_ctrl_after_linearize(DevPlan d) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < d.B) ctrl_after_linearize(d, p);
}

// The same in one CTA, in the body of the iteration loop (a CUDA-graph while
// node): the loop goes on while any problem does and passes are left.  (Every
// iteration of an active problem counts one, so where the control is at the
// end of the body the limit only makes the loop's end explicit.)
__global__ void __launch_bounds__(256) k_ctrl_loop(DevPlan d, LoopControl c) {
  int any = 0;
  for (int p = threadIdx.x; p < d.B; p += blockDim.x) any |= ctrl_after_linearize(d, p);
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    const int passes = ++d.state[0].loop_passes;
    ++d.state[0].loop_total;
    cudaGraphSetConditional(c.handle, any && passes <= c.limit ? 1u : 0u);
  }
}

// The LM step decision of problem p from the back-substitution's partial
// sums (every thread of the CTA takes part; thread 0 decides).  Run by
// k_ctrl_step, or (CG = true) by the last CTA of k_backsub to finish for p.
template <bool CG>
__device__ void ctrl_step_body(const DevPlan& d, int p, double* red) {
  LMState& st = d.state[p];
  if (!st.active) return;
  const bool failed = d.factor_flag[p] != 0;
  double dn2 = 0, xn2 = 0, gd = 0, er = 0;
  if (!failed) {
    double sp[3], si[3];
    prob_sums<3, CG>(d.pt_chunk_sum, 3, d.prob_pt_chunk_off, p, red, sp);
    prob_sums<3, CG>(d.img_chunk_sum, 3, d.prob_img_chunk_off, p, red, si);
    dn2 = sp[0] + si[0];
    xn2 = sp[1] + si[1];
    gd = sp[2] + si[2];
    // PCG leaves the image rows with residual r: the model decrease gains r^T delta_i
    if (d.pcg) er = prob_sum<CG>(d.pcg_part, kPcgSlots, 6, d.prob_ext_chunk_off, p, red);
    if (d.free_cams) {
      double sc[3];
      prob_sums<3, CG>(d.cam_sum, 3, d.prob_cam_off, p, red, sc);
      dn2 += sc[0];
      xn2 += sc[1];
      gd += sc[2];
    }
  }
  if (threadIdx.x != 0) return;
  st.iter += 1;
  st.evaluate = 0;
  if (d.factor_flag[p] == 2) {        // a bounded wait of the factorization ran out
    st.active = 0;
    st.stop = GBA_STOP_ERROR;
    st.status = GBA_ERR_TIMEOUT;
    return;
  }
  // the flag is consumed: cleared here (the next iteration's point factor
  // may run beside the previous linearization's control, so not there)
  d.factor_flag[p] = 0;
  if (failed) {
    st.factor_fail += 1;
    st.rejected += 1;
    st.mu *= st.nu;
    st.nu *= 2.0;
  } else {
    st.dn2 = dn2;
    st.xn2 = xn2;
    st.gd = gd;
    st.er = er;
    if (sqrt(dn2) <= d.eps2 * (sqrt(xn2) + d.eps2)) {
      st.active = 0;
      st.stop = GBA_STOP_SMALL_STEP;
    } else {
      st.evaluate = 1;
    }
  }
}

__global__ void __launch_bounds__(kCtrlThreads) k_ctrl_step(DevPlan d) {
  __shared__ double red[32];
  ctrl_step_body<false>(d, blockIdx.x, red);
}

// The LM accept / reject decision of problem p from the candidate cost's
// partial sums.  Run by k_ctrl_accept, or (CG = true) by the last CTA of the
// candidate cost kernel to finish for p.
template <bool CG>
__device__ void ctrl_accept_body(const DevPlan& d, int p, double* red) {
  LMState& st = d.state[p];
  if (!st.evaluate) return;
  double fr[2];
  prob_sums<2, CG>(d.key_chunk_sum, 2, d.prob_key_chunk_off, p, red, fr);
  if (threadIdx.x != 0) return;
  double Fn = fr[0];
  const double raw_n = fr[1];
  if (d.cons_cost) Fn += d.cons_cost[p];
  st.evaluate = 0;
  st.F_new = Fn;
  // predicted decrease of the quadratic model, 2 g^T d - d^T N d, written
  // with (N + mu I) d = g - e (e = 0 for the exact factorization)
  const double denom = st.mu * st.dn2 + st.gd + st.er;
  const double rho = (st.F - Fn) / denom;
  if (isfinite(Fn) && denom > 0.0 && rho > 0.0) {
    if (d.ftol > 0.0 && st.F - Fn <= d.ftol * st.F) {   // Ceres' function tolerance
      st.active = 0;
      st.stop = GBA_STOP_SMALL_COST_CHANGE;
    }
    st.parity ^= 1;
    st.F = Fn;
    st.raw = raw_n;
    st.relin = 1;
    const double t = 2.0 * rho - 1.0;
    st.mu *= fmax(1.0 / 3.0, 1.0 - t * t * t);
    st.nu = 2.0;
    st.accepted += 1;
    st.ginf_bits = 0ull;
    st.maxdiag_bits = 0ull;
  } else {
    st.mu *= st.nu;
    st.nu *= 2.0;
    st.rejected += 1;
  }
}

__global__ void __launch_bounds__(kCtrlThreads) k_ctrl_accept(DevPlan d) {
  __shared__ double red[32];
  ctrl_accept_body<false>(d, blockIdx.x, red);
}

// The observed keys as double-float pairs (hi = float(v), lo = float(v - hi)).
__global__ void k_split_keys(DevPlan d, float2* out) {
  const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= d.K) return;
  const double2 o = d.key_obs[k];
  out[2 * k] = ff_split(o.x);
  out[2 * k + 1] = ff_split(o.y);
}

// The current x of every problem (each in its own parity; x0 before a run)
// gathered into out = [points 3P][images 6I][cameras 10 Ctot].
__global__ void k_gather_x(DevPlan d, int ran, double* out) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long np = 3LL * d.P, ni = 6LL * d.I, nc = d.free_cams ? 10LL * d.Ctot : 0;
  if (e < np) {
    const int par = d.state[d.pt_prob[e / 3]].parity;
    out[e] = ran ? d.x_pt[par][e] : d.x0_pt[e];
  } else if (e < np + ni) {
    const long long f = e - np;
    const int par = d.state[d.img_prob[f / 6]].parity;
    out[e] = ran ? d.x_img[par][f] : d.x0_img[f];
  } else if (e < np + ni + nc) {
    const long long f = e - np - ni;
    const int par = d.state[d.cam_info[f / 10].z].parity;
    out[e] = ran ? d.x_cam[par][f] : d.x0_cam[f];
  }
}

// ---------------------------------------------------------------------------
// stage outputs for parity checks
// ---------------------------------------------------------------------------
__global__ void k_vector_function(DevPlan d, double* y) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.K) return;
  const int img = d.key_img[k], pt = d.key_pt[k];
  const int par = d.state[d.img_prob[img]].parity;
  double R[12];
  for (int j = 0; j < 12; ++j) R[j] = d.img_rot[par][12LL * img + j];
  const double* xp = d.x_pt[par] + 3LL * pt;
  double X[3] = {xp[0], xp[1], xp[2]};
  double cam[10];
  for (int j = 0; j < 10; ++j) cam[j] = d.cam64[par][10 * d.img_cam[img] + j];
  Proj64 p;
  project64(R, X, cam, p);
  y[2LL * k] = p.u;
  y[2LL * k + 1] = p.v;
}

template <typename T>
__global__ void k_jacobian_out(DevPlan d, double* jp_out, double* ji_out, double* jc_out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.K) return;
  const int img = d.key_img[k], pt = d.key_pt[k];
  const int par = d.state[d.img_prob[img]].parity;
  const double* xp = d.x_pt[par] + 3LL * pt;
  T cam[10];
  load_cam<T>(d, par, d.img_cam[img], cam);
  T jp[6], ji[12], jc[20];
  if constexpr (sizeof(T) == sizeof(double)) {
    double R[12], Jl[9];
    for (int j = 0; j < 12; ++j) R[j] = d.img_rot[par][12LL * img + j];
    for (int j = 0; j < 9; ++j) Jl[j] = tptr<double>(d.img_lin[par])[12LL * img + j];
    Proj64 p;
    project64(R, xp, cam, p);
    jacobian64(R, Jl, cam, p, true, 1.0, 0.0, 1.0, 1.0, jp, ji);
    camera_jacobian64(p, cam, jc);
  } else {
    T nrm[2];
    const T X[3] = {T(xp[0]), T(xp[1]), T(xp[2])};
    T il[12];
    for (int j = 0; j < 12; ++j) il[j] = tptr<T>(d.img_lin[par])[12LL * img + j];
    key_jacobian<T>(X, il, cam, jp, ji, nrm);
    camera_jacobian<T>(nrm[0], nrm[1], cam, jc);
  }
  for (int j = 0; j < 6; ++j) jp_out[6LL * k + j] = double(jp[j]);
  for (int j = 0; j < 12; ++j) ji_out[12LL * k + j] = double(ji[j]);
  if (jc_out) {   // all ten columns; the host keeps the computed ones
    for (int j = 0; j < 20; ++j) jc_out[20LL * k + j] = double(jc[j]);
  }
}

template <typename T>
int run_cholesky_factor(const DevPlan& d, cudaStream_t s) {
  if (d.chol_small) {   // factor and solve in one launch (small systems, FP32)
    if constexpr (sizeof(T) == sizeof(float))
      k_chol_small<T><<<dim3(1u, unsigned(d.B)), kCholSmallThreads, chol_small_smem<T>(d.max_nt), s>>>(d);
    return 1;
  }
  if (d.df_grid > 0) {
    DevPlan dd = d;
    void* args[] = {&dd};
    const cudaError_t e = cudaLaunchCooperativeKernel(
        reinterpret_cast<const void*>(&k_chol_dataflow<T>), dim3(unsigned(d.df_grid)),
        dim3(kDfThreads), args, df_smem_bytes<T>(d.df_max_own), s);
    if (e != cudaSuccess) {
      std::fprintf(stderr, "gba: k_chol_dataflow launch failed: %s\n", cudaGetErrorString(e));
      throw CudaError{GBA_ERR_CUDA};
    }
    return 1;
  }
  int n = 0;
  k_chol_step<T><<<dim3(unsigned(d.max_nt), unsigned(d.B)), 256, 0, s>>>(d, -1);
  ++n;
  for (int k = 0; k + 1 < d.max_nt; ++k) {
    const int Tn = d.max_nt - k - 1;
    k_chol_step<T><<<dim3(unsigned(Tn * (Tn + 1) / 2), unsigned(d.B)), 256, 0, s>>>(d, k);
    ++n;
  }
  return n;
}

template <typename T>
int run_cholesky_solve(const DevPlan& d, cudaStream_t s) {
  if (d.chol_small) return 0;   // done by k_chol_small
  if (d.max_nt <= kSolveSmallTiles)
    k_chol_solve_small<T><<<dim3(1u, unsigned(d.B)), 256, 0, s>>>(d);
  else if (d.solve_drop_step >= 0 || d.solve_spin_limit != kSolveSpin)
    k_chol_solve<T, true><<<dim3(unsigned(kSolveRanks), unsigned(d.B)), 256, solve_smem_bytes<T>(d.max_nt), s>>>(d);
  else
    k_chol_solve<T, false><<<dim3(unsigned(kSolveRanks), unsigned(d.B)), 256, solve_smem_bytes<T>(d.max_nt), s>>>(d);
  return 1;
}

template <typename T>
void run_image_prep(const DevPlan& d, int which, cudaStream_t s) {
  if (d.I > 0) k_image_prep<T><<<(d.I + 127) / 128, 128, 0, s>>>(d, which);
}

}  // namespace

// ===========================================================================
// launchers
// ===========================================================================
#define GBA_DISPATCH(d, KERNEL_CALL)                       \
  do {                                                     \
    if ((d).precision == GBA_PRECISION_MIXED) {            \
      using T = float;                                     \
      KERNEL_CALL;                                         \
    } else {                                               \
      using T = double;                                    \
      KERNEL_CALL;                                         \
    }                                                      \
  } while (0)

int launch_init(const DevPlan& d, cudaStream_t s) {
  k_init<<<(d.B + 127) / 128, 128, 0, s>>>(d);
  long long tot = 3LL * d.P + 6LL * d.I + (d.free_cams ? 10LL * d.Ctot : 0);
  if (tot > 0) {
    k_copy_x0<<<int((tot + 255) / 256), 256, 0, s>>>(d);
    return 2;
  }
  return 1;
}

int launch_image_prep(const DevPlan& d, int which, cudaStream_t s) {
  int n = 0;
  if (d.free_cams && d.Ctot > 0) {
    k_cam_prep<<<(d.Ctot + 127) / 128, 128, 0, s>>>(d, which);
    ++n;
  }
  // the candidate's image rotations come from k_backsub
  if (d.I <= 0 || which == 1) return n;
  GBA_DISPATCH(d, run_image_prep<T>(d, which, s));
  return n + 1;
}

int launch_cost(const DevPlan& d, int which, cudaStream_t s) {
  int n = 0;
  // constraint and prior terms first: the accept decision folded into the
  // key cost kernel adds them
  if (d.n_cons > 0 || d.n_priors > 0) {
    k_cons_cost<<<d.B, 256, 0, s>>>(d, which);
    ++n;
  }
  if (d.n_key_chunks > 0) {
    if (d.precision == GBA_PRECISION_MIXED)
      k_cost_ff<<<d.n_key_chunks, 256, 0, s>>>(d, which);
    else
      k_cost<<<d.n_key_chunks, 256, 0, s>>>(d, which);
    ++n;
  }
  return n;
}

int launch_ctrl_initial_cost(const DevPlan& d, cudaStream_t s) {
  k_ctrl_initial_cost<<<d.B, kCtrlThreads, 0, s>>>(d);
  return 1;
}

int launch_linearize(const DevPlan& d, cudaStream_t s, bool keys) {
  int n = 0;
  if (keys && d.n_key_chunks > 0) {
    GBA_DISPATCH(d, (k_linearize_keys<T><<<d.n_key_chunks, 256, 0, s>>>(d)));
    ++n;
  }
  if (d.n_pt_chunks > 0) {
    GBA_DISPATCH(d, (k_point_reduce<T><<<d.n_pt_chunks, kPointChunk, 0, s>>>(d)));
    ++n;
  }
  return n;
}

int launch_image_reduce(const DevPlan& d, cudaStream_t s) {
  if (d.n_img_items <= 0) return 0;
  GBA_DISPATCH(d, (k_image_reduce<T><<<(d.n_img_items + 7) / 8, 256, 0, s>>>(d)));
  if (d.precision == GBA_PRECISION_MIXED)
    k_image_finalize<float><<<(d.I + 7) / 8, 256, 0, s>>>(d);
  else
    k_image_finalize<double><<<d.I, kFinalizeThreads, 0, s>>>(d);
  if (!d.free_cams) return 2;
  GBA_DISPATCH(d, (k_image_cam_reduce<T><<<d.n_img_items, 128, 0, s>>>(d)));
  k_image_cam_finalize<<<d.I, kImgCamVals, 0, s>>>(d);
  k_cam_finalize<<<d.Ctot, kImgCamVals * kCamGroups, 0, s>>>(d);
  return 5;
}

int launch_ctrl_after_linearize(const DevPlan& d, cudaStream_t s, const LoopControl* loop) {
  if (loop) {
    k_ctrl_loop<<<1, 256, 0, s>>>(d, *loop);
    return 1;
  }
  k_ctrl_after_linearize<<<(d.B + 127) / 128, 128, 0, s>>>(d);
  return 1;
}

int launch_z_slots(const DevPlan& d, int* key_slot, cudaStream_t s) {
  int n = 0;
  if (d.K > 0) {
    k_key_slots<<<(d.K + 255) / 256, 256, 0, s>>>(d.img_keys, d.K, key_slot);
    ++n;
  }
  if (d.n_items > 0) {
    k_pairs_to_slots<<<(d.n_items + 3) / 4, 128, 0, s>>>(d.items, d.n_items, d.blk_ij, key_slot, d.K,
                                                        const_cast<int2*>(d.pairs));
    ++n;
  }
  return n;
}

int launch_point_schur(const DevPlan& d, cudaStream_t s) {
  int n = 0;
  if (d.n_pt_chunks > 0) {
    GBA_DISPATCH(d, (k_point_factor<T><<<d.n_pt_chunks, kPointChunk, 0, s>>>(d)));
    ++n;
  }
  if (d.n_key_chunks > 0) {
    GBA_DISPATCH(d, (k_key_z<T><<<d.n_key_chunks * d.key_z_split, 256, 0, s>>>(d)));
    ++n;
  }
  if (d.free_cams && d.R > 0) {
    GBA_DISPATCH(d, (k_camrec_z<T><<<d.n_pt_chunks, kPointChunk, 0, s>>>(d)));
    ++n;
  }
  return n;
}

int launch_assemble_items(const DevPlan& d, cudaStream_t s) {
  if (d.n_items <= 0) return 0;
  GBA_DISPATCH(d, (k_assemble_items<T><<<(d.n_items + 3) / 4, 128, 0, s>>>(d, d.n_items)));
  return 1;
}

int launch_assemble_S(const DevPlan& d, cudaStream_t s) {
  if (d.max_n <= 0) return 0;
  if (d.blk_prob && d.n_blocks > 0) {
    const size_t tsz = d.precision == GBA_PRECISION_MIXED ? sizeof(float) : sizeof(double);
    if (!d.s_complete && cudaMemsetAsync(d.S, 0, size_t(d.s_elems) * tsz, s) != cudaSuccess)
      throw CudaError{GBA_ERR_CUDA};
    const unsigned g = unsigned((36LL * d.n_blocks + 255) / 256);
    GBA_DISPATCH(d, (k_assemble_S_blocks<T><<<g, 256, 0, s>>>(d)));
    return 1;
  }
  dim3 grid(unsigned((1LL * d.max_n * d.max_n + 255) / 256), unsigned(d.B));
  GBA_DISPATCH(d, (k_assemble_S<T><<<grid, 256, 0, s>>>(d)));
  return 1;
}

int launch_assemble(const DevPlan& d, cudaStream_t s) {
  return launch_assemble_items(d, s) + launch_assemble_S(d, s);
}

int launch_cholesky_factor(const DevPlan& d, cudaStream_t s) {
  if (d.max_nt <= 0) return 0;
  int n = 0;
  GBA_DISPATCH(d, n = run_cholesky_factor<T>(d, s));
  return n;
}

// Allows a kernel all the dynamic shared memory its static arrays leave of the
// device's limit (the limit is the function's, shared by every plan, so it is
// never set to one plan's need); false when `need` bytes do not fit.
static bool allow_dynamic_smem(const void* fn, size_t need) {
  cudaFuncAttributes a = {};
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&a, fn) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  const long long most = (long long)optin - (long long)a.sharedSizeBytes;
  if ((long long)need > most) return false;
  if (a.maxDynamicSharedSizeBytes < most &&
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(most)) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

int prepare_cholesky_solve(int max_nt, int precision) {
  if (max_nt <= kSolveSmallTiles) return GBA_OK;
  const bool mixed = precision == GBA_PRECISION_MIXED;
  const size_t bytes = mixed ? solve_smem_bytes<float>(max_nt) : solve_smem_bytes<double>(max_nt);
  if (bytes <= 48 * 1024) return GBA_OK;
  const void* f[2] = {mixed ? reinterpret_cast<const void*>(&k_chol_solve<float, false>)
                            : reinterpret_cast<const void*>(&k_chol_solve<double, false>),
                      mixed ? reinterpret_cast<const void*>(&k_chol_solve<float, true>)
                            : reinterpret_cast<const void*>(&k_chol_solve<double, true>)};
  for (const void* fn : f)
    if (!allow_dynamic_smem(fn, bytes)) return GBA_ERR_UNSUPPORTED;
  return GBA_OK;
}

bool prepare_chol_small(int max_nt, int precision) {
  if (precision != GBA_PRECISION_MIXED || max_nt < 1 || max_nt > kSolveSmallTiles) return false;
  return allow_dynamic_smem(reinterpret_cast<const void*>(&k_chol_small<float>), chol_small_smem<float>(max_nt));
}

int launch_cholesky_solve(const DevPlan& d, cudaStream_t s) {
  if (d.max_nt <= 0) return 0;
  int n = 0;
  GBA_DISPATCH(d, n = run_cholesky_solve<T>(d, s));
  return n;
}

template <typename T>
bool dataflow_layout_t(int nt, int device, int* grid, int* max_own, int* rows, int* helpers,
                       std::vector<int>* own_off,
                       std::vector<int2>* own) {
  int sms = 0, coop = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (!coop || nt < 2) return false;
  const DfLayout l = df_layout(nt, sizeof(T) == sizeof(float), sms);
  const int G = l.grid, mo = l.max_own;
  const size_t smem = df_smem_bytes<T>(mo);
  if (mo > (l.rows > 0 ? kDfWorkerTiles : kDfThreads) ||
      !allow_dynamic_smem(reinterpret_cast<const void*>(&k_chol_dataflow<T>), smem))
    return false;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chol_dataflow<T>, kDfThreads, smem) !=
          cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    return false;
  }
  own_off->assign(1, 0);
  own->clear();
  for (const auto& o : l.own) {
    for (const DfTile& t : o) own->push_back(make_int2(t.i, t.j));
    own_off->push_back(int(own->size()));
  }
  *grid = G;
  *max_own = mo;
  *rows = l.rows;
  *helpers = l.helpers;
  return true;
}

bool dataflow_layout(int nt, bool mixed, int device, int* grid, int* max_own, int* rows, int* helpers,
                     std::vector<int>* own_off, std::vector<int2>* own) {
  return mixed ? dataflow_layout_t<float>(nt, device, grid, max_own, rows, helpers, own_off, own)
               : dataflow_layout_t<double>(nt, device, grid, max_own, rows, helpers, own_off, own);
}

int launch_assemble_blocks(const DevPlan& d, cudaStream_t s) {
  if (d.n_blocks <= 0) return 0;
  const long long n = 36LL * d.n_blocks;
  GBA_DISPATCH(d, (k_assemble_blocks<T><<<unsigned((n + 255) / 256), 256, 0, s>>>(d)));
  return 1;
}

int launch_pcg_setup(const DevPlan& d, cudaStream_t s) {
  if (d.I_ext <= 0) return 0;
  GBA_DISPATCH(d, (k_pcg_precond<T><<<(d.I_ext + 127) / 128, 128, 0, s>>>(d)));
  GBA_DISPATCH(d, (k_pcg_init<T><<<d.n_ext_chunks, 256, 0, s>>>(d)));
  return 2;
}

int launch_pcg_iterations(const DevPlan& d, cudaStream_t s, bool nested) {
  if (d.I_ext <= 0) return 0;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (d.pcg_it && d.pcg_body_stream && cudaStreamIsCapturing(s, &cs) == cudaSuccess &&
      cs == cudaStreamCaptureStatusActive) {
    // in a CUDA graph: a while node whose body runs two iterations and the
    // loop control, so the iterations after convergence are not launched
    cudaGraph_t g = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    cudaGraphConditionalHandle h = 0;
    cudaGraphNodeParams cp = {};
    cudaGraphNode_t node = nullptr;
    if (cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, nullptr, &nd) != cudaSuccess ||
        cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault) != cudaSuccess)
      throw CudaError{GBA_ERR_CUDA};
    if (nested) {
      k_pcg_loop_open<<<1, 1, 0, s>>>(h);
      if (cudaStreamGetCaptureInfo(s, &cs, nullptr, &g, &deps, nullptr, &nd) != cudaSuccess)
        throw CudaError{GBA_ERR_CUDA};
    }
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if (cudaGraphAddNode(&node, g, deps, nullptr, nd, &cp) != cudaSuccess) throw CudaError{GBA_ERR_CUDA};
    cudaStream_t bs = d.pcg_body_stream;
    if (cudaStreamBeginCaptureToGraph(bs, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                      cudaStreamCaptureModeThreadLocal) != cudaSuccess)
      throw CudaError{GBA_ERR_CUDA};
    for (int u = 0; u < 2; ++u) {
      GBA_DISPATCH(d, (k_pcg_spmv<T><<<d.n_ext_chunks, 256, 0, bs>>>(d, u, 1)));
      GBA_DISPATCH(d, (k_pcg_update<T><<<d.n_ext_chunks, 256, 0, bs>>>(d, u, 1)));
    }
    k_pcg_loop_ctrl<<<1, 32, 0, bs>>>(d, h);
    cudaGraph_t body = nullptr;
    if (cudaStreamEndCapture(bs, &body) != cudaSuccess ||
        cudaStreamUpdateCaptureDependencies(s, &node, nullptr, 1, cudaStreamSetCaptureDependencies) != cudaSuccess)
      throw CudaError{GBA_ERR_CUDA};
    return nested ? 6 : 5;   // (one pass of the body; it runs as many passes as the solve needs)
  }
  for (int it = 0; it < d.pcg_max_iterations; ++it) {
    GBA_DISPATCH(d, (k_pcg_spmv<T><<<d.n_ext_chunks, 256, 0, s>>>(d, it, 0)));
    GBA_DISPATCH(d, (k_pcg_update<T><<<d.n_ext_chunks, 256, 0, s>>>(d, it, 0)));
  }
  return 2 * d.pcg_max_iterations;
}

int launch_cholesky(const DevPlan& d, cudaStream_t s) {
  return launch_cholesky_factor(d, s) + launch_cholesky_solve(d, s);
}

int launch_backsub(const DevPlan& d, cudaStream_t s) {
  const int g = d.n_pt_chunks + d.n_img_chunks;
  if (g <= 0) return 0;
  int n = 0;
  // the cameras' step first: with the control folded into k_backsub, its
  // last CTA reads the cameras' partial sums too
  if (d.free_cams && d.Ctot > 0) {
    GBA_DISPATCH(d, (k_cam_backsub<T><<<(d.Ctot + 127) / 128, 128, 0, s>>>(d)));
    ++n;
  }
  GBA_DISPATCH(d, (k_backsub<T><<<g, kPointChunk, 0, s>>>(d)));
  return n + 1;
}

int launch_ctrl_step(const DevPlan& d, cudaStream_t s) {
  if (d.fold_ctrl) return 0;   // done by the last CTA of each problem in k_backsub
  k_ctrl_step<<<d.B, kCtrlThreads, 0, s>>>(d);
  return 1;
}

int launch_ctrl_accept(const DevPlan& d, cudaStream_t s) {
  if (d.fold_ctrl) return 0;   // done by the last CTA of each problem in the candidate cost
  k_ctrl_accept<<<d.B, kCtrlThreads, 0, s>>>(d);
  return 1;
}

int launch_vector_function(const DevPlan& d, double* y, cudaStream_t s) {
  if (d.K <= 0) return 0;
  k_vector_function<<<(d.K + 255) / 256, 256, 0, s>>>(d, y);
  return 1;
}

int launch_split_keys(const DevPlan& d, float2* out, cudaStream_t s) {
  if (d.K <= 0) return 0;
  k_split_keys<<<unsigned((d.K + 255) / 256), 256, 0, s>>>(d, out);
  return 1;
}

int launch_gather_x(const DevPlan& d, int ran, double* out, cudaStream_t s) {
  const long long n = 3LL * d.P + 6LL * d.I + (d.free_cams ? 10LL * d.Ctot : 0);
  if (n <= 0) return 0;
  k_gather_x<<<unsigned((n + 255) / 256), 256, 0, s>>>(d, ran, out);
  return 1;
}

int launch_jacobian_out(const DevPlan& d, double* jp, double* ji, double* jc, cudaStream_t s) {
  if (d.K <= 0) return 0;
  GBA_DISPATCH(d, (k_jacobian_out<T><<<(d.K + 255) / 256, 256, 0, s>>>(d, jp, ji, jc)));
  return 1;
}

// ===========================================================================
// Key pairs of the Schur complement built on the device (plans without free
// cameras).  Problem q's image pairs (a, c), a <= c local images, have the
// codes first_code(q) + a * Ie + c; the problems' code ranges follow each
// other, so code order is the host's block order of the concatenated plan.
// The device counts the pairs of every code (atomics), marks the blocks
// (codes with pairs, and every diagonal), numbers them and their first pairs
// by exclusive scans, and returns the block list.  Every point then writes
// its pairs (a <= c over its keys, point-major) with their block id, and a
// stable LSD radix sort by block id leaves each block's pairs in point order
// -- the same list, in the same order, as the host build's placement.
// Problem records pinfo[q] = (first image, Ie, first code, 0).
// ===========================================================================
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortPerThread = 8;
constexpr int kSortTile = kSortThreads * kSortPerThread;   // elements per tile
constexpr int kScanChunk = 4096;                             // per scan CTA (1024 x 4)
constexpr int kScanTop = 8192;                               // chunk totals one CTA scans

// Pairs per code: one thread per point, one atomic per key pair (keys of a
// point are in image order).
__global__ void __launch_bounds__(128) k_count_pairs(int P, const int* __restrict__ pt_key_off,
                                                     const int* __restrict__ key_img,
                                                     const int* __restrict__ pt_prob,
                                                     const int4* __restrict__ pinfo, int* __restrict__ cnt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P) return;
  const int4 pq = pinfo[pt_prob[i]];
  const int k0 = pt_key_off[i], k1 = pt_key_off[i + 1];
  for (int a = k0; a < k1; ++a) {
    const long long row = pq.z + (long long)(key_img[a] - pq.x) * pq.y;
    for (int c = a; c < k1; ++c) atomicAdd(cnt + row + (key_img[c] - pq.x), 1);
  }
}

// Pairs of each point, k (k + 1) / 2; entry P is 0 (the scan makes it the total).
__global__ void __launch_bounds__(256) k_point_pairs(int P, const int* __restrict__ pt_key_off,
                                                     int* __restrict__ pp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > P) return;
  int v = 0;
  if (i < P) {
    const int k = pt_key_off[i + 1] - pt_key_off[i];
    v = k * (k + 1) / 2;
  }
  pp[i] = v;
}

// A block for every image pair a < c with pairs and for every diagonal
// (a == c, even without keys).
__device__ __forceinline__ bool block_present(int local, int Ie, int count) {
  const int a = local / Ie, c = local - a * Ie;
  return a == c || (c > a && count > 0);
}

// grid (codes of the largest problem / 256, problems)
__global__ void __launch_bounds__(256) k_block_marks(const int4* __restrict__ pinfo, const int* __restrict__ cnt,
                                                     int* __restrict__ mark, int* __restrict__ off) {
  const int4 pq = pinfo[blockIdx.y];
  const int local = blockIdx.x * blockDim.x + threadIdx.x;
  if (local >= pq.y * pq.y) return;
  const int e = pq.z + local;
  const int v = cnt[e];
  mark[e] = block_present(local, pq.y, v) ? 1 : 0;
  off[e] = v;
}

// After the scans: bid[e] = the block id (or -1); the block list (local
// code, first pair) in block order; each problem's first block (its block
// (0, 0) is always present); info = (blocks, pairs) from the last code of
// problem qlast (the last with images: its block (Ie-1, Ie-1)).
__global__ void __launch_bounds__(256) k_block_lists(const int4* __restrict__ pinfo, int qlast,
                                                     const int* __restrict__ cnt, int* __restrict__ bid,
                                                     const int* __restrict__ off, int* __restrict__ blk_code,
                                                     int* __restrict__ blk_first, int* __restrict__ prob_block,
                                                     int* __restrict__ info) {
  const int q = blockIdx.y;
  const int4 pq = pinfo[q];
  const int local = blockIdx.x * blockDim.x + threadIdx.x;
  const int L = pq.y * pq.y;
  if (local >= L) return;
  const int e = pq.z + local;
  const int v = cnt[e];
  const bool m = block_present(local, pq.y, v);
  const int b = bid[e];
  if (m) {
    blk_code[b] = local;
    blk_first[b] = off[e];
  }
  bid[e] = m ? b : -1;
  if (local == 0) prob_block[q] = b;
  if (q == qlast && local == L - 1) {
    info[0] = b + 1;
    info[1] = off[e] + v;
  }
}

__global__ void __launch_bounds__(128) k_enumerate_pairs(int P, const int* __restrict__ pt_key_off,
                                                         const int* __restrict__ key_img,
                                                         const int* __restrict__ pt_prob,
                                                         const int4* __restrict__ pinfo,
                                                         const int* __restrict__ pp_off,
                                                         const int* __restrict__ bid, int* __restrict__ keys,
                                                         int2* __restrict__ vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P) return;
  const int4 pq = pinfo[pt_prob[i]];
  const int k0 = pt_key_off[i], k1 = pt_key_off[i + 1];
  int pos = pp_off[i];
  for (int a = k0; a < k1; ++a) {
    const long long row = pq.z + (long long)(key_img[a] - pq.x) * pq.y;
    for (int c = a; c < k1; ++c, ++pos) {
      keys[pos] = bid[row + (key_img[c] - pq.x)];
      // a pair of a diagonal block is a key with itself: carry its point instead
      vals[pos] = make_int2(a, a == c ? i : c);
    }
  }
}

// Per tile, the count of each 8-bit digit of the keys (digit-major output).
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const int* __restrict__ keys, long long n, int shift,
                                                               int ntiles, int* __restrict__ hist) {
  __shared__ int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long t0 = (long long)blockIdx.x * kSortTile;
#pragma unroll
  for (int j = 0; j < kSortPerThread; ++j) {
    const long long e = t0 + (long long)j * kSortThreads + threadIdx.x;
    if (e < n) atomicAdd(&h[(keys[e] >> shift) & 255], 1);
  }
  __syncthreads();
  hist[(long long)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of v [n] in chunks of kScanChunk: each CTA scans its chunk
// and writes the chunk total to sums.
__global__ void __launch_bounds__(1024) k_scan_chunks(int* __restrict__ v, long long n, int* __restrict__ sums) {
  __shared__ int wsum[32];
  const long long base = (long long)blockIdx.x * kScanChunk + 4LL * threadIdx.x;
  int x[4], t = 0;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    x[u] = base + u < n ? v[base + u] : 0;
    t += x[u];
  }
  // inclusive scan of the thread totals across the CTA
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int inc = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) wsum[w] = inc;
  __syncthreads();
  if (w == 0) {
    int ws = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += y;
    }
    wsum[lane] = ws;   // inclusive over warps
  }
  __syncthreads();
  int run = inc - t + (w > 0 ? wsum[w - 1] : 0);   // exclusive prefix of this thread
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (base + u < n) v[base + u] = run;
    run += x[u];
  }
  if (threadIdx.x == 1023) sums[blockIdx.x] = run;
}

// Exclusive scan of the chunk totals (at most 8192) in one CTA.
__global__ void __launch_bounds__(1024) k_scan_totals(int* __restrict__ sums, int m) {
  __shared__ int part[1024];
  const int per = (m + 1023) / 1024;
  const int b = threadIdx.x * per;
  int t = 0;
  for (int u = 0; u < per; ++u)
    if (b + u < m) t += sums[b + u];
  part[threadIdx.x] = t;
  __syncthreads();
  if (threadIdx.x == 0) {   // 1024 values: serial in one thread, fixed order
    int run = 0;
    for (int u = 0; u < 1024; ++u) {
      const int y = part[u];
      part[u] = run;
      run += y;
    }
  }
  __syncthreads();
  int run = part[threadIdx.x];
  for (int u = 0; u < per; ++u)
    if (b + u < m) {
      const int y = sums[b + u];
      sums[b + u] = run;
      run += y;
    }
}

__global__ void __launch_bounds__(1024) k_scan_add(int* __restrict__ v, long long n, const int* __restrict__ sums) {
  const long long base = (long long)blockIdx.x * kScanChunk + 4LL * threadIdx.x;
  const int add = sums[blockIdx.x];
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (base + u < n) v[base + u] += add;
}

// Stable scatter of one tile by the digit at `shift`: elements are ranked in
// tile order (256 at a time, warp by warp, lane by lane).  A position outside
// [0, n) is not written and raises *bad.
__global__ void __launch_bounds__(kSortThreads) k_radix_scatter(const int* __restrict__ keys,
                                                                  const int2* __restrict__ vals, long long n,
                                                                  int shift, int ntiles,
                                                                  const int* __restrict__ offs,
                                                                  int* __restrict__ okeys,
                                                                  int2* __restrict__ ovals, int* bad) {
  __shared__ int base[256], run[256], wc[kSortThreads / 32][256];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  base[t] = offs[(long long)t * ntiles + blockIdx.x];
  run[t] = 0;
  const long long t0 = (long long)blockIdx.x * kSortTile;
  for (int j = 0; j < kSortPerThread; ++j) {
#pragma unroll
    for (int ww = 0; ww < kSortThreads / 32; ++ww) wc[ww][t] = 0;
    __syncthreads();
    const long long e = t0 + (long long)j * kSortThreads + t;
    const bool valid = e < n;
    const int key = valid ? keys[e] : 0;
    const int dgt = valid ? (key >> shift) & 255 : 256;
    const unsigned peers = __match_any_sync(0xffffffffu, dgt);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (valid && rank == 0) wc[w][dgt] = __popc(peers);
    __syncthreads();
    if (valid) {
      int pos = base[dgt] + run[dgt] + rank;
      for (int ww = 0; ww < w; ++ww) pos += wc[ww][dgt];
      if (pos >= 0 && (long long)pos < n) {
        okeys[pos] = key;
        ovals[pos] = vals[e];
      } else {
        atomicExch(bad, 1);
      }
    }
    __syncthreads();
    int add = 0;
#pragma unroll
    for (int ww = 0; ww < kSortThreads / 32; ++ww) add += wc[ww][t];
    run[t] += add;
    __syncthreads();
  }
}

// Exclusive scan of v [L] in place: chunks of kScanChunk, their totals
// scanned the same way (one CTA once there are at most kScanTop of them).
// scratch holds scan_scratch_ints(L) ints.
int scan_exclusive(int* v, long long L, int* scratch, cudaStream_t s) {
  if (L <= 0) return 0;
  const long long nchunks = (L + kScanChunk - 1) / kScanChunk;
  k_scan_chunks<<<unsigned(nchunks), 1024, 0, s>>>(v, L, scratch);
  int n = 1;
  if (nchunks <= kScanTop) {
    k_scan_totals<<<1, 1024, 0, s>>>(scratch, int(nchunks));
    ++n;
  } else {
    n += scan_exclusive(scratch, nchunks, scratch + nchunks, s);
  }
  k_scan_add<<<unsigned(nchunks), 1024, 0, s>>>(v, L, scratch);
  return n + 1;
}

}  // namespace

long long scan_scratch_ints(long long L) {
  long long t = 0;
  while (L > 0) {
    const long long c = (L + kScanChunk - 1) / kScanChunk;
    t += c;
    if (c <= kScanTop) break;
    L = c;
  }
  return std::max<long long>(t, 1);
}

int count_blocks_on_device(int nprob, int qlast, int max_ie, int P, const int4* d_pinfo, const int* d_pt_key_off,
                           const int* d_key_img, const int* d_pt_prob, long long L, int* d_cnt, int* d_bid,
                           int* d_off, int* d_scratch, int* d_blk_code, int* d_blk_first, int* d_prob_block,
                           int* d_info, cudaStream_t s) {
  int launches = 0;
  if (L <= 0 || nprob <= 0 || nprob > 65535) return -1;
  if (cudaMemsetAsync(d_cnt, 0, sizeof(int) * size_t(L), s) != cudaSuccess) return -1;
  if (P > 0) {
    k_count_pairs<<<unsigned((P + 127) / 128), 128, 0, s>>>(P, d_pt_key_off, d_key_img, d_pt_prob, d_pinfo, d_cnt);
    ++launches;
  }
  const dim3 g(unsigned(((long long)max_ie * max_ie + 255) / 256), unsigned(nprob));
  k_block_marks<<<g, 256, 0, s>>>(d_pinfo, d_cnt, d_bid, d_off);
  launches += 1 + scan_exclusive(d_bid, L, d_scratch, s) + scan_exclusive(d_off, L, d_scratch, s);
  k_block_lists<<<g, 256, 0, s>>>(d_pinfo, qlast, d_cnt, d_bid, d_off, d_blk_code, d_blk_first, d_prob_block,
                                  d_info);
  return launches + 1;
}

int build_pairs_on_device(int P, int nblocks, const int4* d_pinfo, const int* d_pt_key_off, const int* d_key_img,
                          const int* d_pt_prob, int* d_pp, const int* d_bid, long long n, int* d_keys0,
                          int2* d_vals0, int* d_keys1, int2* d_vals1, int* d_hist, int* d_scratch, int* d_bad,
                          int2** out, cudaStream_t s) {
  int launches = 0;
  if (P > 0) {
    k_point_pairs<<<unsigned((P + 256) / 256), 256, 0, s>>>(P, d_pt_key_off, d_pp);
    launches += 1 + scan_exclusive(d_pp, (long long)P + 1, d_scratch, s);
    k_enumerate_pairs<<<unsigned((P + 127) / 128), 128, 0, s>>>(P, d_pt_key_off, d_key_img, d_pt_prob, d_pinfo,
                                                                  d_pp, d_bid, d_keys0, d_vals0);
    ++launches;
  }
  int bits = 1;
  while (bits < 31 && (1LL << bits) < nblocks) ++bits;
  const int passes = (bits + 7) / 8;
  const int ntiles = int((n + kSortTile - 1) / kSortTile);
  const long long L = 256LL * ntiles;
  int* kin = d_keys0;
  int2* vin = d_vals0;
  int* kout = d_keys1;
  int2* vout = d_vals1;
  for (int pass = 0; pass < passes && n > 0; ++pass) {
    const int shift = 8 * pass;
    k_radix_hist<<<unsigned(ntiles), kSortThreads, 0, s>>>(kin, n, shift, ntiles, d_hist);
    launches += 2 + scan_exclusive(d_hist, L, d_scratch, s);
    k_radix_scatter<<<unsigned(ntiles), kSortThreads, 0, s>>>(kin, vin, n, shift, ntiles, d_hist, kout, vout,
                                                              d_bad);
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  *out = vin;
  return launches;
}

void pairs_sort_scratch(long long n, int P, long long* hist_ints, long long* scratch_ints) {
  const long long ntiles = (n + kSortTile - 1) / kSortTile;
  *hist_ints = 256LL * std::max<long long>(ntiles, 1);
  *scratch_ints = std::max(scan_scratch_ints(*hist_ints), scan_scratch_ints((long long)P + 1));
}

}  // namespace gba
