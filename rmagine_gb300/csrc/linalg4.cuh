// The Umeyama step's 3x3 problems with four lanes each, for a whole warp at once:
// singular value decomposition, the Kabsch/Umeyama rotation, the rotation-matrix
// -> quaternion conversion, and the rotation's derivative.
//
// Replaces umeyama_transform (optimization.cpp:12-49, linalg.cu:1157-1200).
//
// A binary64 instruction takes a warp of the GB300 64 cycles, whether one of its
// lanes is on or all 32, and a solve by one thread has 400 of them.  So the lanes
// of a group of four hold a column each (the fourth repeats the third), products
// of matrices cost a third, and what need not be exact is done in binary32:
//
//   * the eigenvectors of A = C^T C to binary32, by Jacobi sweeps;
//   * that frame made a rotation in binary64 through its quaternion (a rotation
//     matrix formed from a quaternion and divided by its norm is orthogonal);
//   * A in that frame, whose off-diagonal elements are at most some 1e-6, and one
//     step of perturbation theory to second order: the frame is turned by the
//     antisymmetric X with X_ij = a_ij / (a_jj - a_ii) and by the correction that
//     is left of a_ij.  The angles are binary32 numbers, what they leave of a_ij
//     is formed exactly, so that the result is good to binary64.
//
// Where that does not hold (elements out of range, eigenvalues closer than the
// step allows, a rank below two) the group takes svd3_rot, each lane for itself.
// 400 problems (transform alone): 26 us by one thread each, now 10; 40,000: 70,
// which the binary64 pipe bounds.
// All lanes of the warp must call these functions together.
#pragma once

#include "linalg.cuh"

namespace rmg {

__device__ __forceinline__ double pick(int j, double a, double b, double c) { return j == 0 ? a : (j == 1 ? b : c); }

// x of lane i of this lane's group of four.
template <class T>
__device__ __forceinline__ T of4(T x, int i) { return __shfl_sync(0xffffffffu, x, i, 4); }

__device__ __forceinline__ int column4() { return min((int)(threadIdx.x & 3), 2); }

// The frame of all columns from the lanes'.
__device__ __forceinline__ M3d gather4(const double col[3]) {
  M3d m;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) m.a[k][c] = of4(col[k], c);
  return m;
}

// Column `j` of x y and of x y^T, for y's column j or row j.
__device__ __forceinline__ void mul_col(const M3d& x, const double y[3], double r[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) r[i] = x.a[i][0] * y[0] + x.a[i][1] * y[1] + x.a[i][2] * y[2];
}

__device__ __forceinline__ void row_of(const M3d& m, int j, double r[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) r[k] = pick(j, m.a[0][k], m.a[1][k], m.a[2][k]);
}

__device__ __forceinline__ double dot(const double x[3], const double y[3]) {
  return x[0] * y[0] + x[1] * y[1] + x[2] * y[2];
}

// A Jacobi rotation in binary32 for elements of at most 2.
__device__ __forceinline__ void jacobi_rotate_f(float& app, float& aqq, float& apq, float& arp, float& arq, float vp[3],
                                                float vq[3]) {
  if (fabsf(apq) <= 1e-18f) return;
  const float d = aqq - app, h = d * d + 4.0f * apq * apq;
  const float t = __fdividef(2.0f * apq, d + copysignf(h * rsqrtf(h), d));
  const float c = rsqrtf(t * t + 1.0f), s = t * c;
  app -= t * apq;
  aqq += t * apq;
  apq = 0.0f;
  const float x = arp, y = arq;
  arp = c * x - s * y;
  arq = s * x + c * y;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float vx = vp[k], vy = vq[k];
    vp[k] = c * vx - s * vy;
    vq[k] = s * vx + c * vy;
  }
}

// Unit quaternion (x, y, z, w) of the rotation with columns w0, w1, w2, to binary32.
__device__ __forceinline__ void quat_f(const float w0[3], const float w1[3], const float w2[3], float q[4]) {
  const float x = w1[2] - w2[1], y = w2[0] - w0[2], z = w0[1] - w1[0];
  const float xy = w0[1] + w1[0], xz = w0[2] + w2[0], yz = w1[2] + w2[1];
  const float tr = w0[0] + w1[1] + w2[2];
  if (tr > 0.0f) { q[0] = x; q[1] = y; q[2] = z; q[3] = 1.0f + tr; }
  else if (w0[0] > w1[1] && w0[0] > w2[2]) { q[0] = 1.0f + w0[0] - w1[1] - w2[2]; q[1] = xy; q[2] = xz; q[3] = x; }
  else if (w1[1] > w2[2]) { q[0] = xy; q[1] = 1.0f + w1[1] - w0[0] - w2[2]; q[2] = yz; q[3] = y; }
  else { q[0] = xz; q[1] = yz; q[2] = 1.0f + w2[2] - w0[0] - w1[1]; q[3] = z; }
  const float r = rsqrtf(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) q[k] *= r;
}

// Whether any lane of this lane's group is in a warp's vote.
__device__ __forceinline__ bool any4(uint32_t vote) { return (vote >> (threadIdx.x & 28) & 15u) != 0; }

__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }

// svd3_rot of the same C in the four lanes of a group; U, s and V in all of them.
// True if the whole warp's are zero (U and V the identity then).
// Where A = C^T C is diagonal (no correspondences, one, a line along an axis) its
// frame is the identity and needs no pass, which a warp of such problems leaves
// out, and svd3_rot's choices for a rank of one and zero are made here: svd3_rot
// itself takes eight problems to a warp here, where one thread each has 32.
// 40,000 zero matrices (transform alone) 91 -> 19 us, one thread each 37; of rank
// one along an axis 111 -> 51, one thread each 51 (of 400,000 989 -> 444 and 332).
__device__ __forceinline__ bool svd3_lanes(const M3d& C, M3d& U, double s[3], M3d& V) {
  const int j = column4(), n1 = j == 2 ? 0 : j + 1, n2 = 3 - j - n1;
  // column j of A, times the power of two that brings its largest diagonal element to [1, 2)
  double a[3];
  {
    const double cj[3] = {pick(j, C.a[0][0], C.a[0][1], C.a[0][2]), pick(j, C.a[1][0], C.a[1][1], C.a[1][2]),
                          pick(j, C.a[2][0], C.a[2][1], C.a[2][2])};
#pragma unroll
    for (int i = 0; i < 3; ++i) a[i] = C.a[0][i] * cj[0] + C.a[1][i] * cj[1] + C.a[2][i] * cj[2];
  }
  int e = __double2hiint(pick(j, a[0], a[1], a[2])) & 0x7ff00000;
  e = max(max(of4(e, 0), of4(e, 1)), of4(e, 2));
  // (no exchange inside a choice: every lane of the warp takes part in all of them)
  const uint32_t mixed = __ballot_sync(0xffffffffu, !is_zero(pick(j, a[1], a[2], a[0])) || !is_zero(pick(j, a[2], a[0], a[1])));
  const uint32_t some = __ballot_sync(0xffffffffu, !is_zero(pick(j, a[0], a[1], a[2])));
  const bool diagonal = !any4(mixed), zero = !any4(mixed | some);
  uint32_t groups = mixed | mixed >> 1;
  groups |= groups >> 2;
  const bool plain = (groups & 0x11111111u) == 0x11111111u;  // none of the warp's is diagonal
  if (!plain && (mixed | some) == 0) {
    U = V = m3_eye();
    s[0] = s[1] = s[2] = 0.0;
    return true;
  }
  bool bad = !zero && (e < (64 << 20) || e > (1983 << 20));  // (NaN and infinity have the largest exponent)
  const double scale = __hiloint2double(bad || zero ? 0x3ff00000 : (2046 << 20) - e, 0);
#pragma unroll
  for (int i = 0; i < 3; ++i) a[i] *= scale;

  const double a00 = of4(a[0], 0), a01 = of4(a[0], 1), a02 = of4(a[0], 2);
  const double a11 = of4(a[1], 1), a12 = of4(a[1], 2), a22 = of4(a[2], 2);
  float f00 = (float)a00, f01 = (float)a01, f02 = (float)a02, f11 = (float)a11, f12 = (float)a12, f22 = (float)a22;
  double v[3] = {0.0, 0.0, 0.0}, y[3], z[3];  // this lane's column of V, the columns n1 and n2
  double d, off, g;         // elements (j, j) and (j, n1) of A in V's frame, and the gap of their eigenvalues
  float X, fg;
  // One pass, and up to two more for the groups with small eigenvalues closer than a
  // first binary32 frame tells apart: A in that frame is graded, and the next
  // frame's binary32 angles are good relative to those eigenvalues.  The warp's
  // other groups keep their frame meanwhile and form the same numbers from it again,
  // so that a problem's result does not depend on its neighbours.
  bool again = true;
#pragma unroll 1
  for (int pass = 0; mixed != 0; ++pass) {
    float w0[3] = {1.f, 0.f, 0.f}, w1[3] = {0.f, 1.f, 0.f}, w2[3] = {0.f, 0.f, 1.f};
    const float tol = pass == 0 ? 1e-13f : 1e-34f;
#pragma unroll 1
    for (int sweep = 0; sweep < 6 && f01 * f01 + f02 * f02 + f12 * f12 > tol; ++sweep) {
      jacobi_rotate_f(f00, f11, f01, f02, f12, w0, w1);
      jacobi_rotate_f(f00, f22, f02, f01, f12, w0, w2);
      jacobi_rotate_f(f11, f22, f12, f01, f02, w1, w2);
    }
    float q[4];
    quat_f(w0, w1, w2, q);
    const double qj = j == 0 ? q[0] : (j == 1 ? q[1] : q[2]), q1 = j == 0 ? q[1] : (j == 1 ? q[2] : q[0]),
                 q2 = j == 0 ? q[2] : (j == 1 ? q[0] : q[1]), w = q[3];
    const double p = w * w + qj * qj, m = q1 * q1 + q2 * q2, e1 = (p + m) - 1.0;
    const double inv = 1.0 - e1 * (1.0 - e1 * (1.0 - e1)), inv2 = inv + inv;  // 1 / |q|^2, e1 ~ 1e-7
    const double rj = (p - m) * inv, r1 = (qj * q1 + w * q2) * inv2, r2 = (qj * q2 - w * q1) * inv2;
    const double r[3] = {pick(j, rj, r2, r1), pick(j, r1, rj, r2), pick(j, r2, r1, rj)};
    if (pass == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = r[k];
    } else {
      const M3d old = gather4(v);
      double turned[3];
      mul_col(old, r, turned);
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] = again ? turned[k] : v[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) { y[k] = of4(v[k], n1); z[k] = of4(v[k], n2); }
    const double x[3] = {a00 * v[0] + a01 * v[1] + a02 * v[2], a01 * v[0] + a11 * v[1] + a12 * v[2],
                         a02 * v[0] + a12 * v[1] + a22 * v[2]};
    d = dot(v, x);
    off = dot(y, x);
    g = of4(d, n1) - d;
    fg = (float)g;
    const float fo = (float)off;
    X = fo == 0.0f ? 0.0f : fo / fg;  // X_(j, n1)
    bool far = !(fabsf(X) < 4e-6f);   // third-order terms up to here are below binary64's rounding
    // Equal eigenvalues, diagonal to binary64's rounding of A.  Leaving `off` turns the
    // rotation sought by off / (2 d); small eigenvalues get their frames first (singular
    // values 1, 1e-7, 1e-7 left at once: mean error 8.7e-4, so 2.7e-4, by one thread 3.4e-4).
    if (far && fabsf(fo) <= 4e-16f && (__double2hiint(d) >= 0x3f800000 || pass == 2)) {  // d >= 2^-7
      far = false;
      X = 0.0f;
    }
    const uint32_t away = __ballot_sync(0xffffffffu, far && !bad && !diagonal);
    again = any4(away);
    if (pass == 2 || away == 0) {
      bad = bad || (far && !diagonal);
      break;
    }
    const float fd = (float)d;
    f00 = of4(fd, 0); f11 = of4(fd, 1); f22 = of4(fd, 2);
    f01 = of4(fo, 0); f12 = of4(fo, 1); f02 = of4(fo, 2);
    if (!again) f01 = f12 = f02 = 0.0f;
  }
  if (mixed != 0) {
    const float Xa = of4(X, n1), Xb = of4(X, n2), ga = of4(fg, n1), gb = of4(fg, n2);
    const float rest = (float)(off - g * (double)X) + 0.5f * Xa * Xb * (ga - gb);
    const float Xc = fabsf(rest) <= 4e-16f && !(fabsf(rest) < 1e-8f * fabsf(fg)) ? 0.0f : rest / fg;
    bad = bad || (!(fabsf(Xc) < 1e-8f) && !diagonal);
    const float Xcb = of4(Xc, n2);
    const double p0 = -0.5f * (X * X + Xb * Xb), p1 = (double)(0.5f * Xa * Xb - Xc) - (double)X,
                 p2 = (double)(0.5f * Xa * X + Xcb) + (double)Xb;
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] += p0 * v[k] + p1 * y[k] + p2 * z[k];
  }
  if (!plain && diagonal) {
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = k == j ? 1.0 : 0.0;
  }
  // B = C V: columns s_i u_i; the columns in the order of their lengths, V right-handed
  double B[3];
  mul_col(C, v, B);
  double q = dot(B, B);
  {
    const long long own = __double_as_longlong(q), o1 = of4(own, n1), o2 = of4(own, n2);  // q >= 0: ordered as integers
    const int rank = (o1 > own || (o1 == own && n1 < j)) + (o2 > own || (o2 == own && n2 < j));
    const int r0 = of4(rank, 0), r1 = of4(rank, 1);
    const int src = r0 == j ? 0 : (r1 == j ? 1 : 2);
    const bool odd = r1 != (r0 == 2 ? 0 : r0 + 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      v[k] = of4(v[k], src);
      B[k] = of4(B[k], src);
      if (odd && j == 2) { v[k] = -v[k]; B[k] = -B[k]; }
    }
    q = of4(q, src);
  }
  V = gather4(v);
  const double q0 = of4(q, 0);
  double u0[3], u1[3], u2[3];
  const double i0 = rsqrt(q0);
#pragma unroll
  for (int k = 0; k < 3; ++k) u0[k] = of4(B[k], 0) * i0;
#pragma unroll
  for (int k = 0; k < 3; ++k) u1[k] = of4(B[k], 1);
  const double d01 = dot(u0, u1);
#pragma unroll
  for (int k = 0; k < 3; ++k) u1[k] -= d01 * u0[k];
  double q1 = dot(u1, u1);
  const bool flat = !(q1 > 1e-24 * q0);
  bad = bad || (flat && !diagonal);
  if (!plain) {
    if (flat && diagonal) {  // rank one: any unit vector orthogonal to u0
      const int k = (fabs(u0[0]) <= fabs(u0[1]) && fabs(u0[0]) <= fabs(u0[2])) ? 0 : (fabs(u0[1]) <= fabs(u0[2]) ? 1 : 2);
      const double u0k = pick(k, u0[0], u0[1], u0[2]);
#pragma unroll
      for (int i = 0; i < 3; ++i) u1[i] = (i == k ? 1.0 : 0.0) - u0k * u0[i];
      q1 = dot(u1, u1);
    }
  }
  const double i1 = rsqrt(q1);
#pragma unroll
  for (int k = 0; k < 3; ++k) u1[k] *= i1;
  const double x = pick(j, u0[1], u0[2], u0[0]) * pick(j, u1[2], u1[0], u1[1]) -
                   pick(j, u0[2], u0[0], u0[1]) * pick(j, u1[1], u1[2], u1[0]);
#pragma unroll
  for (int k = 0; k < 3; ++k) u2[k] = of4(x, k);
  const double uj[3] = {pick(j, u0[0], u1[0], u2[0]), pick(j, u0[1], u1[1], u2[1]), pick(j, u0[2], u1[2], u2[2])};
  const double sj = dot(uj, B);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    U.a[k][0] = u0[k]; U.a[k][1] = u1[k]; U.a[k][2] = u2[k];
    s[k] = of4(sj, k);
  }
  if (any4(__ballot_sync(0xffffffffu, bad))) svd3_rot(C, U, s, V);
  if (!plain && zero) {
    U = V;
    s[0] = s[1] = s[2] = 0.0;
  }
  return false;
}

// R = U V^T in all lanes.
__device__ __forceinline__ M3d rotation_lanes(const M3d& U, const M3d& V) {
  double vr[3], r[3];
  row_of(V, column4(), vr);
  mul_col(U, vr, r);
  return gather4(r);
}

// Rotation matrix -> unit quaternion (x, y, z, w), in all lanes.  Branch choice as
// in rmagine's Matrix -> Quaternion cast (math/types/MatrixOps.tcc:1492-1529), so
// both pick the same of the two signs q / -q.
__device__ __forceinline__ void rot_to_quat_lanes(const M3d& R, double q[4]) {
  const int j = column4();
  // lane j: R_21 -+ R_12, R_02 -+ R_20, R_10 -+ R_01
  const double a = pick(j, R.a[2][1], R.a[0][2], R.a[1][0]), b = pick(j, R.a[1][2], R.a[2][0], R.a[0][1]);
  const double minus = a - b, plus = a + b;
  const double x = of4(minus, 0), y = of4(minus, 1), z = of4(minus, 2);
  const double yz = of4(plus, 0), xz = of4(plus, 1), xy = of4(plus, 2);
  const double r0 = R.a[0][0], r1 = R.a[1][1], r2 = R.a[2][2];
  const int big = r0 + r1 + r2 > 0.0 ? 3 : (r0 > r1 && r0 > r2) ? 0 : (r1 > r2 ? 1 : 2);
  // S^2 / 4
  const double arg = (big == 3 ? r0 : big == 0 ? r0 : -r0) + (big == 3 || big == 1 ? r1 : -r1) +
                     (big == 3 || big == 2 ? r2 : -r2) + 1.0;
  const double h = rsqrt(arg), rS = 0.5 * h, c = arg * rS;  // 1 / S and S / 4
  q[0] = big == 0 ? c : (big == 3 ? x : big == 1 ? xy : xz) * rS;
  q[1] = big == 1 ? c : (big == 3 ? y : big == 0 ? xy : yz) * rS;
  q[2] = big == 2 ? c : (big == 3 ? z : big == 0 ? xz : yz) * rS;
  q[3] = big == 3 ? c : (big == 0 ? x : big == 1 ? y : z) * rS;
  const double n = rsqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2] + q[3] * q[3]);
#pragma unroll
  for (int k = 0; k < 4; ++k) q[k] *= n;
}

// Umeyama / Kabsch of the same problem in the four lanes of a group: R = U V^T,
// t = m - R d, in all of them.  n == 0 or a non-finite result gives the identity
// rotation (optimization.cpp:19-46).
__device__ __forceinline__ void umeyama_lanes(const M3d& C, const double d[3], const double m[3], unsigned int n,
                                              double q[4], double t[3]) {
  M3d U, V;
  double s[3];
  M3d R = m3_eye();
  bool identity = svd3_lanes(C, U, s, V);
  if (!identity) {  // the whole warp's
    R = rotation_lanes(U, V);
    rot_to_quat_lanes(R, q);
    identity = n == 0 || !(isfinite(q[0]) && isfinite(q[1]) && isfinite(q[2]) && isfinite(q[3]));
  }
  if (identity) {
    R = m3_eye();
    q[0] = q[1] = q[2] = 0.0; q[3] = 1.0;
  }
  const int j = column4();
  double r[3];
  row_of(R, j, r);
  const double x = pick(j, m[0], m[1], m[2]) - dot(r, d);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double tk = of4(x, k);  // every lane of the warp takes part, whatever its own n
    t[k] = n == 0 ? 0.0 : tk;
  }
}

// Gradient of L through R = U V^T (C = U diag(s) V^T, rotations U, V):
// dL/dC = U K V^T with K_ij = (G_ij - G_ji) / (s_i + s_j) for i != j, K_ii = 0,
// G = U^T (dL/dR) V.  Where s_i + s_j <= kRotGradGap * s0 the optimal rotation
// about the axis u_i x u_j is not unique (collinear correspondences: s2 = s3 = 0;
// a reflection with two equal singular values: s2 = -s3) and R is not
// differentiable there: that pair contributes no gradient (K_ij = K_ji = 0).
// The rest of the gradient is exact; close to the boundary it grows like
// 1 / (s_i + s_j), as the rotation's true derivative does.
//
// This lane's column j of it, given column j of dL/dR.
__device__ __forceinline__ void rotation_backward_lanes(const M3d& U, const double s[3], const M3d& V,
                                                        const double gR[3], double out[3]) {
  const int j = column4(), n1 = j == 2 ? 0 : j + 1;
  // H = U^T gR, then column j of G = H V
  double h[3], vj[3], G[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) h[i] = U.a[0][i] * gR[0] + U.a[1][i] * gR[1] + U.a[2][i] * gR[2];
  const M3d H = gather4(h);
#pragma unroll
  for (int k = 0; k < 3; ++k) vj[k] = pick(j, V.a[k][0], V.a[k][1], V.a[k][2]);
  mul_col(H, vj, G);
  // K_(j, n1) = (G_(j, n1) - G_(n1, j)) / (s_j + s_n1)
  const double g0 = of4(G[0], n1), g1 = of4(G[1], n1), g2 = of4(G[2], n1);
  const double up = pick(j, g0, g1, g2), low = pick(n1, G[0], G[1], G[2]);
  const double den = pick(j, s[0], s[1], s[2]) + pick(n1, s[0], s[1], s[2]);
  const double kj = den > kRotGradGap * fabs(s[0]) ? (up - low) / den : 0.0;
  const double k01 = of4(kj, 0), k12 = of4(kj, 1), k20 = of4(kj, 2);
  // U K V^T: column j of (K V^T) first
  double vr[3];
  row_of(V, j, vr);
  const double y[3] = {k01 * vr[1] - k20 * vr[2], k12 * vr[2] - k01 * vr[0], k20 * vr[0] - k12 * vr[1]};
  mul_col(U, y, out);
}

}  // namespace rmg
