// Binary64 3x3 singular value decomposition with right-handed factors by one
// thread (linalg4.cuh solves the Umeyama step with four lanes per problem).
//
// Replaces rmagine's Numerical-Recipes svdcmp (src/rmagine_core/src/math/
// linalg.cpp:101, device src/rmagine_cuda/src/math/linalg.cu:61) and
// umeyama_transform (optimization.cpp:12-49, linalg.cu:1157-1200).
//
// SVD: cyclic Jacobi eigen-decomposition of the symmetric A = C^T C gives V
// and sigma^2 (sorted descending, V made right-handed); U = [u1, u2, u1 x u2]
// with u1, u2 from C V by Gram-Schmidt, and the third singular value carries
// the sign: sigma3 = u3 . (C v3).  With U and V both rotations,
// C = U diag(s1, s2, s3) V^T and the Umeyama rotation (R = U S V^T with the
// reflection fix S = diag(1, 1, sign det(U V^T)) of the usual SVD) is simply
// R = U V^T.
#pragma once

#include <math.h>

namespace rmg {

struct M3d { double a[3][3]; };  // row-major

__host__ __device__ inline M3d m3_zero() {
  M3d r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r.a[i][j] = 0.0;
  return r;
}

__host__ __device__ inline M3d m3_eye() {
  M3d r = m3_zero();
  r.a[0][0] = r.a[1][1] = r.a[2][2] = 1.0;
  return r;
}

__host__ __device__ inline M3d m3_mul(const M3d& x, const M3d& y) {
  M3d r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r.a[i][j] = x.a[i][0] * y.a[0][j] + x.a[i][1] * y.a[1][j] + x.a[i][2] * y.a[2][j];
  return r;
}

__host__ __device__ inline M3d m3_mul_tn(const M3d& x, const M3d& y) {  // x^T y
  M3d r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r.a[i][j] = x.a[0][i] * y.a[0][j] + x.a[1][i] * y.a[1][j] + x.a[2][i] * y.a[2][j];
  return r;
}

__host__ __device__ inline double m3_det(const M3d& m) {
  return m.a[0][0] * (m.a[1][1] * m.a[2][2] - m.a[1][2] * m.a[2][1]) -
         m.a[0][1] * (m.a[1][0] * m.a[2][2] - m.a[1][2] * m.a[2][0]) +
         m.a[0][2] * (m.a[1][0] * m.a[2][1] - m.a[1][1] * m.a[2][0]);
}

__host__ __device__ inline double rsqrt_d(double x) {
#ifdef __CUDA_ARCH__
  return rsqrt(x);
#else
  return 1.0 / sqrt(x);
#endif
}

// One Jacobi rotation of a symmetric 3x3 matrix on its axes p and q (r the
// third): zeroes apq, V <- V J.  Everything stays in registers, and the chain
// has three long operations (square root, division, reciprocal square root):
// t = 2 apq / (d + sign(d) sqrt(d^2 + 4 apq^2)), d = aqq - app.  (An angle found
// in binary32 with a binary64 normalisation measured slower: conversions and
// one sweep more.)
__host__ __device__ inline void jacobi_rotate(double& app, double& aqq, double& apq, double& arp, double& arq,
                                              double vp[3], double vq[3]) {
  if (fabs(apq) <= 1e-300) return;
  const double d = aqq - app;
  const double t = 2.0 * apq / (d + copysign(sqrt(d * d + 4.0 * apq * apq), d));
  const double c = rsqrt_d(t * t + 1.0), s = t * c;
  app -= t * apq;
  aqq += t * apq;
  apq = 0.0;
  const double x = arp, y = arq;
  arp = c * x - s * y;
  arq = s * x + c * y;
  for (int k = 0; k < 3; ++k) {
    const double vx = vp[k], vy = vq[k];
    vp[k] = c * vx - s * vy;
    vq[k] = s * vx + c * vy;
  }
}

__host__ __device__ inline void swap_columns(double& lx, double& ly, double x[3], double y[3]) {
  if (!(lx < ly)) return;
  double t = lx; lx = ly; ly = t;
  for (int k = 0; k < 3; ++k) { t = x[k]; x[k] = y[k]; y[k] = t; }
}

// C = U diag(s) V^T with U, V proper rotations; s[0] >= s[1] >= |s[2]|, s[2] signed.
//
// One thread solves one matrix, so what counts is the length of its binary64
// chain.  400 matrices: 41 us with indexed arrays in local memory, five
// divisions and square roots per rotation and four warps to an SM's narrow
// binary64 pipe; 26 us in registers, with three, one warp to a CTA.
__host__ __device__ inline void svd3_rot(const M3d& C, M3d& U, double s[3], M3d& V) {
  const M3d A = m3_mul_tn(C, C);
  double a00 = A.a[0][0], a11 = A.a[1][1], a22 = A.a[2][2], a01 = A.a[0][1], a02 = A.a[0][2], a12 = A.a[1][2];
  double v0[3] = {1.0, 0.0, 0.0}, v1[3] = {0.0, 1.0, 0.0}, v2[3] = {0.0, 0.0, 1.0};  // columns of V
  const double scale = fmax(fmax(fmax(fabs(a00), fabs(a11)), fmax(fabs(a22), fabs(a01))), fmax(fabs(a02), fabs(a12)));
  if (scale > 0.0) {
    for (int sweep = 0; sweep < 24; ++sweep) {
      const double off = a01 * a01 + a02 * a02 + a12 * a12;
      if (off <= 1e-36 * scale * scale) break;
      jacobi_rotate(a00, a11, a01, a02, a12, v0, v1);
      jacobi_rotate(a00, a22, a02, a01, a12, v0, v2);
      jacobi_rotate(a11, a22, a12, a01, a02, v1, v2);
    }
  }
  // eigenvalues descending
  swap_columns(a00, a11, v0, v1);
  swap_columns(a11, a22, v1, v2);
  swap_columns(a00, a11, v0, v1);
  for (int k = 0; k < 3; ++k) { V.a[k][0] = v0[k]; V.a[k][1] = v1[k]; V.a[k][2] = v2[k]; }
  if (m3_det(V) < 0.0)
    for (int k = 0; k < 3; ++k) V.a[k][2] = -V.a[k][2];
  // B = C V: columns b_i = s_i u_i
  const M3d B = m3_mul(C, V);
  double u1[3] = {B.a[0][0], B.a[1][0], B.a[2][0]};
  double n1 = sqrt(u1[0] * u1[0] + u1[1] * u1[1] + u1[2] * u1[2]);
  if (!(n1 > 1e-300)) {  // C == 0: any frame, take V's
    U = V;
    s[0] = s[1] = s[2] = 0.0;
    return;
  }
  const double r1 = 1.0 / n1;
  for (int k = 0; k < 3; ++k) u1[k] *= r1;
  double u2[3] = {B.a[0][1], B.a[1][1], B.a[2][1]};
  double d12 = u1[0] * u2[0] + u1[1] * u2[1] + u1[2] * u2[2];
  for (int k = 0; k < 3; ++k) u2[k] -= d12 * u1[k];
  double n2 = sqrt(u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2]);
  if (!(n2 > 1e-12 * n1)) {  // rank 1: any unit vector orthogonal to u1
    const int k = (fabs(u1[0]) <= fabs(u1[1]) && fabs(u1[0]) <= fabs(u1[2])) ? 0 : (fabs(u1[1]) <= fabs(u1[2]) ? 1 : 2);
    d12 = k == 0 ? u1[0] : (k == 1 ? u1[1] : u1[2]);
    for (int j = 0; j < 3; ++j) u2[j] = (j == k ? 1.0 : 0.0) - d12 * u1[j];
    n2 = sqrt(u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2]);
  }
  const double r2 = 1.0 / n2;
  for (int k = 0; k < 3; ++k) u2[k] *= r2;
  const double u3[3] = {u1[1] * u2[2] - u1[2] * u2[1], u1[2] * u2[0] - u1[0] * u2[2], u1[0] * u2[1] - u1[1] * u2[0]};
  for (int k = 0; k < 3; ++k) { U.a[k][0] = u1[k]; U.a[k][1] = u2[k]; U.a[k][2] = u3[k]; }
  s[0] = n1;
  s[1] = u2[0] * B.a[0][1] + u2[1] * B.a[1][1] + u2[2] * B.a[2][1];
  s[2] = u3[0] * B.a[0][2] + u3[1] * B.a[1][2] + u3[2] * B.a[2][2];
}

// Relative size below which s_i + s_j counts as zero in the rotation's gradient.
// The covariance reaches the backward in binary32 (rmagine's CrossStatistics),
// so singular values carry an absolute error of about 1e-7 s0: a smaller sum
// is rounding noise, and dividing by it would only amplify that noise.
constexpr double kRotGradGap = 1e-6;

}  // namespace rmg
