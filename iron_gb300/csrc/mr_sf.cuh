// mr_sf.cuh -- sum-factorised FP64 element operations of the Q2/Q1 Mooney-Rivlin element.
//
// GB300's FP64 pipe issues one warp instruction in 64 cycles, so the FP64 kernels of the element
// cost what they issue on it.  The triquadratic basis on the 3x3x3 Gauss rule is a tensor product,
// so gradients at the Gauss points and their transposes are taken one xi direction at a time, a
// line of three values per thread: about 350 FP64 operations a field where the dense tables
// (27 points x 3 derivatives x 27 nodes) take 2,187.
//
// On one line with nodes at 0, 1/2, 1 and Gauss points 1/2 - t, 1/2, 1/2 + t (t = sqrt(0.6) / 2):
//   u(x) = u1 + b (x - 1/2) + 2 c (x - 1/2)^2,   b = u2 - u0,   c = u0 - 2 u1 + u2.
// b and c are formed from the node differences u1 - u0 and u2 - u1, which are exact for coordinates
// of neighbouring nodes, so the derivatives carry less rounding than the dense sums.
//
// Index conventions: 27-entry blocks are xi1 fastest; thread j < 27 of an element owns Gauss point j
// in the point phases and line j in the transform stages.
#pragma once

#include "gfe_internal.cuh"

namespace mr_sf {

constexpr double kT = 0.38729833462074168852;   // sqrt(0.6) / 2
constexpr double k4T = 4.0 * kT;
constexpr double k8T = 8.0 * kT;

__device__ __forceinline__ double point_weight(int g) {
  const double we = 5.0 / 18.0, wm = 8.0 / 18.0;
  return (g % 3 == 1 ? wm : we) * ((g / 3) % 3 == 1 ? wm : we) * (g / 9 == 1 ? wm : we);
}

// values and derivatives of one line at its three Gauss points
__device__ __forceinline__ void line_val(double u0, double u1, double u2, double (&v)[3]) {
  const double e1 = u1 - u0, e2 = u2 - u1, b = e1 + e2, c = e2 - e1;
  const double m = fma(0.3, c, u1);
  v[0] = fma(-kT, b, m);
  v[1] = u1;
  v[2] = fma(kT, b, m);
}
__device__ __forceinline__ void line_der(double u0, double u1, double u2, double (&d)[3]) {
  const double e1 = u1 - u0, e2 = u2 - u1, b = e1 + e2, c = e2 - e1;
  d[0] = fma(-k4T, c, b);
  d[1] = b;
  d[2] = fma(k4T, c, b);
}
__device__ __forceinline__ void line_val_der(double u0, double u1, double u2, double (&v)[3], double (&d)[3]) {
  const double e1 = u1 - u0, e2 = u2 - u1, b = e1 + e2, c = e2 - e1;
  const double m = fma(0.3, c, u1);
  v[0] = fma(-kT, b, m);
  v[1] = u1;
  v[2] = fma(kT, b, m);
  d[0] = fma(-k4T, c, b);
  d[1] = b;
  d[2] = fma(k4T, c, b);
}
// transposes: o[a] = sum_g r_g (value, derivative) of the node functions a
__device__ __forceinline__ void line_val_t(double r0, double r1, double r2, double (&o)[3]) {
  const double s = r0 + r2, q = r2 - r0, a = 0.3 * s;
  o[0] = fma(-kT, q, a);
  o[1] = fma(0.4, s, r1);
  o[2] = fma(kT, q, a);
}
__device__ __forceinline__ void line_der_t(double r0, double r1, double r2, double (&o)[3]) {
  const double q = r2 - r0, t = r0 + r2 + r1;
  o[0] = fma(k4T, q, -t);
  o[1] = -k8T * q;
  o[2] = fma(k4T, q, t);
}
// line_der_t of r plus line_val_t of s
__device__ __forceinline__ void line_der_val_t(double r0, double r1, double r2, double s0, double s1, double s2,
                                               double (&o)[3]) {
  const double q = r2 - r0, t = r0 + r2 + r1;
  const double ss = s0 + s2, sq = s2 - s0;
  const double a = 0.3 * ss, bq = fma(kT, sq, t);
  const double e = fma(k4T, q, a);
  o[0] = e - bq;
  o[1] = fma(-k8T, q, fma(0.4, ss, s1));
  o[2] = e + bq;
}
// transpose of the linear (pressure) line: o[0] with 1 - x, o[1] with x
__device__ __forceinline__ void line_lin_t(double r0, double r1, double r2, double (&o)[2]) {
  const double h = 0.5 * (r0 + r2 + r1), q = r2 - r0;
  o[0] = fma(-kT, q, h);
  o[1] = fma(kT, q, h);
}

// Gradients of one three-component field: thread j < 27 of the element, node values u[c * 27 + n],
// scratch A[162], B[243]; the caller's barrier SYNC separates the stages and precedes the call and
// the first read of the result grad[(c * 3 + k) * 27 + g] (which may be the memory of u and A).
template <typename Sync>
__device__ __forceinline__ void field_gradients(int j, bool on, const double* u, double* A, double* B, double* grad,
                                                Sync sync) {
  const int f = j / 9, r = j % 9, hi = r / 3, lo = r % 3;
  if (on) {  // xi1: line (component f, n3 = hi, n2 = lo)
    const double* s = u + f * 27 + r * 3;
    double v[3], d[3];
    line_val_der(s[0], s[1], s[2], v, d);
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      A[f * 27 + r * 3 + g] = v[g];
      A[81 + f * 27 + r * 3 + g] = d[g];
    }
  }
  sync();
  if (on) {  // xi2: line (f, n3 = hi, g1 = lo)
    const double* s = A + f * 27 + hi * 9 + lo;
    double v[3], d[3], w[3];
    line_val_der(s[0], s[3], s[6], v, d);
    line_val(s[81], s[84], s[87], w);
    double* o = B + f * 27 + hi * 9 + lo;
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      o[g * 3] = v[g];
      o[81 + g * 3] = d[g];
      o[162 + g * 3] = w[g];
    }
  }
  sync();
  if (on) {  // xi3: line (f, g2 = hi, g1 = lo)
    const double* s = B + f * 27 + r;
    double d1[3], d2[3], d3[3];
    line_val(s[162], s[171], s[180], d1);
    line_val(s[81], s[90], s[99], d2);
    line_der(s[0], s[9], s[18], d3);
    double* o = grad + f * 81 + r;
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      o[g * 9] = d1[g];
      o[27 + g * 9] = d2[g];
      o[54 + g * 9] = d3[g];
    }
  }
}

// Transpose of field_gradients: point values P[(k * 3 + c) * 27 + g] (derivative direction k, component
// c) to out(c * 27 + n, value); scratch A[243], which may not overlap P, and B (162 words) which may be P's
// memory.  Barriers as above.
template <typename Sync, typename Out>
__device__ __forceinline__ void field_gradients_t(int j, bool on, const double* P, double* A, double* B, Sync sync,
                                                  Out out) {
  const int f = j / 9, r = j % 9, hi = r / 3, lo = r % 3;
  if (on) {  // xi3: line (f, g2 = hi, g1 = lo)
    const double* s = P + f * 27 + r;
    double a1[3], a2[3], a3[3];
    line_val_t(s[0], s[9], s[18], a1);
    line_val_t(s[81], s[90], s[99], a2);
    line_der_t(s[162], s[171], s[180], a3);
    double* o = A + f * 27 + r;
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      o[n * 9] = a1[n];
      o[81 + n * 9] = a2[n];
      o[162 + n * 9] = a3[n];
    }
  }
  sync();
  if (on) {  // xi2: line (f, n3 = hi, g1 = lo)
    const double* s = A + f * 27 + hi * 9 + lo;
    double b1[3], b23[3];
    line_val_t(s[0], s[3], s[6], b1);
    line_der_val_t(s[81], s[84], s[87], s[162], s[165], s[168], b23);
    double* o = B + f * 27 + hi * 9 + lo;
#pragma unroll
    for (int n = 0; n < 3; ++n) {
      o[n * 3] = b1[n];
      o[81 + n * 3] = b23[n];
    }
  }
  sync();
  if (on) {  // xi1: line (f, n3 = hi, n2 = lo)
    const double* s = B + f * 27 + r * 3;
    double o[3];
    line_der_val_t(s[0], s[1], s[2], s[81], s[82], s[83], o);
#pragma unroll
    for (int n = 0; n < 3; ++n) out(f * 27 + r * 3 + n, o[n]);
  }
}

// Transpose of the pressure interpolation: point values q[27] to out(b, value), b < 8; the stages run
// between the same barriers as field_gradients_t's.  S1[18], S2[12] scratch.
__device__ __forceinline__ void pressure_t_stage3(int j, const double* q, double* S1) {
  if (j < 9) {
    double o[2];
    line_lin_t(q[j], q[9 + j], q[18 + j], o);
    S1[j] = o[0];
    S1[9 + j] = o[1];
  }
}
__device__ __forceinline__ void pressure_t_stage2(int j, const double* S1, double* S2) {
  if (j < 6) {  // (n3 = j / 3, g1 = j % 3)
    const double* s = S1 + (j / 3) * 9 + j % 3;
    double o[2];
    line_lin_t(s[0], s[3], s[6], o);
    S2[(j / 3) * 6 + j % 3] = o[0];
    S2[(j / 3) * 6 + 3 + j % 3] = o[1];
  }
}
template <typename Out>
__device__ __forceinline__ void pressure_t_stage1(int j, const double* S2, Out out) {
  if (j < 4) {  // (n3, n2)
    const double* s = S2 + j * 3;
    double o[2];
    line_lin_t(s[0], s[1], s[2], o);
    out(j * 2, o[0]);
    out(j * 2 + 1, o[1]);
  }
}

// pressure at Gauss point g from the 8 corner values
__device__ __forceinline__ double point_pressure(int g, const double* p) {
  const double x1 = g % 3 == 0 ? 0.5 - kT : (g % 3 == 1 ? 0.5 : 0.5 + kT);
  const double x2 = (g / 3) % 3 == 0 ? 0.5 - kT : ((g / 3) % 3 == 1 ? 0.5 : 0.5 + kT);
  const double x3 = g / 9 == 0 ? 0.5 - kT : (g / 9 == 1 ? 0.5 : 0.5 + kT);
  const double a00 = fma(x1, p[1] - p[0], p[0]), a10 = fma(x1, p[3] - p[2], p[2]);
  const double a01 = fma(x1, p[5] - p[4], p[4]), a11 = fma(x1, p[7] - p[6], p[6]);
  const double b0 = fma(x2, a10 - a00, a00), b1 = fma(x2, a11 - a01, a01);
  return fma(x3, b1 - b0, b0);
}

// ---- point formulas -----------------------------------------------------------------------------
// With Z = dz/dxi, X = dx/dxi and Iron's fibre-free material frame A = (N^T X)^-1, N the columns of X
// normalised (src/coordinate_routines.F90:3841-3947), the residual's Cauchy stress
// (src/finite_elasticity_routines.F90:6985-7061) depends on F = Z A only through F F^T = Z H Z^T with
// H = A A^T: six numbers a point (geometry below).  With
// J = J_z / J_x, r = J^(-1/3) and B = r^2 Z H Z^T,
//   sigma = dev((t1 B^2 + t2 B) / J) + p I,  t1 = -2 c2,  t2 = 2 (c1 + tr(B) c2),
// and the first Piola form of the residual is P[xi][m] = w J_z (Z^-1 sigma)[xi][m] =
// w sign(det Z) sum_c cof[c][xi] sigma[c][m] with the cofactors cof of Z: no division.
// Symmetric 3x3 matrices are packed 00 11 22 01 02 12.

// cofactors by cross products of the rows of Z[c][k]; returns the determinant
__device__ __forceinline__ double cofactors(const double (&Z)[3][3], double (&cof)[3][3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int a = (c + 1) % 3, b = (c + 2) % 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
      cof[c][k] = Z[a][k1] * Z[b][k2] - Z[a][k2] * Z[b][k1];
    }
  }
  return Z[0][0] * cof[0][0] + Z[0][1] * cof[0][1] + Z[0][2] * cof[0][2];
}

// Factor of the reference metric and J_x of a reference gradient matrix X.  H = A A^T with A = (N^T X)^-1 and
// N^T X = D^-1/2 G (G = X^T X, D = diag G), so K = H^-1 = G D^-1 G is the Gram matrix of G's columns in the weights
// 1/D: orthogonalising them gives K = U^T diag(d) U with U unit upper triangular, and
//   Z H Z^T = V diag(e) V^T,  V = Z U^-1,  e = 1 / d,      h = u01 u02 u12 e0 e1 e2,
// without a square root.  V is found by substitution and never multiplies out H: K has the fourth power of X's
// condition, and inverting it, or forming Z H Z^T from any H, cancels that many digits.  Relative error of the stress
// term P at a point of an element sheared by 3 (10) in two planes: 3e-14 (3e-12), as with Iron's own order of
// operations; with H = (G D^-1 G)^-1 5e-12 (6e-8), with H = G^-1 D G^-1 1e-12 (1e-8).  On a box U is the identity and
// e0, e1, e2 differ by the rounding of a product or two: near the undeformed state the deviator amplifies differences
// between B's diagonal entries, so the diagonal is formed as G_kk r^2 plus small terms.
__device__ __forceinline__ double geometry(const double (&X)[3][3], double (&h)[6]) {
  double G[6];
#pragma unroll
  for (int i = 0; i < 3; ++i) G[i] = X[0][i] * X[0][i] + X[1][i] * X[1][i] + X[2][i] * X[2][i];
  G[3] = X[0][0] * X[0][1] + X[1][0] * X[1][1] + X[2][0] * X[2][1];
  G[4] = X[0][0] * X[0][2] + X[1][0] * X[1][2] + X[2][0] * X[2][2];
  G[5] = X[0][1] * X[0][2] + X[1][1] * X[1][2] + X[2][1] * X[2][2];
  const double g01 = G[0] * G[1], d = 1.0 / (g01 * G[2]);
  const double i0 = G[1] * G[2] * d, i1 = G[0] * G[2] * d, i2 = g01 * d;  // 1 / G_kk
  // first column (G00, G01, G02), weighted (1, w1, w2)
  const double w1 = G[3] * i1, w2 = G[4] * i2;
  h[3] = 1.0 / (G[0] + fma(G[3], w1, G[4] * w2));
  h[0] = fma(2.0, G[3], w2 * G[5]) * h[3];
  h[1] = fma(2.0, G[4], w1 * G[5]) * h[3];
  // the others less their part along it: (a0, G11 ra, a2), (b0, b1, G22 rb)
  const double a0 = fma(-h[0], G[0], G[3]), ra = fma(-h[0], w1, 1.0), a2 = fma(-h[0], G[4], G[5]);
  const double b0 = fma(-h[1], G[0], G[4]), b1 = fma(-h[1], G[3], G[5]), rb = fma(-h[1], w2, 1.0);
  const double a0i = a0 * i0, a2i = a2 * i2;
  h[4] = 1.0 / fma(G[1] * ra, ra, fma(a0, a0i, a2 * a2i));
  h[2] = fma(a0i, b0, fma(ra, b1, a2 * rb)) * h[4];
  // the third less its part along the second: (c0, c1, G22 rc)
  const double c0 = fma(-h[2], a0, b0), c1 = fma(-h[2], G[1] * ra, b1), rc = fma(-h[2], a2i, rb);
  h[5] = 1.0 / fma(G[2] * rc, rc, fma(c0 * i0, c0, c1 * i1 * c1));
  return fabs(X[0][0] * (X[1][1] * X[2][2] - X[1][2] * X[2][1]) + X[0][1] * (X[1][2] * X[2][0] - X[1][0] * X[2][2]) +
              X[0][2] * (X[1][0] * X[2][1] - X[1][1] * X[2][0]));
}

// row of V = Z U^-1
__device__ __forceinline__ void row_v(const double (&z)[3], const double (&h)[6], double (&v)[3]) {
  v[0] = z[0];
  v[1] = fma(-v[0], h[0], z[1]);
  v[2] = fma(-v[0], h[1], fma(-v[1], h[2], z[2]));
}
// row of V diag(e)
__device__ __forceinline__ void row_e(const double (&v)[3], const double (&h)[6], double (&y)[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) y[k] = v[k] * h[3 + k];
}
// row of Z H = V diag(e) U^-T from the row of V diag(e)
__device__ __forceinline__ void row_zh(const double (&y)[3], const double (&h)[6], double (&w)[3]) {
  w[2] = y[2];
  w[1] = fma(-h[2], w[2], y[1]);
  w[0] = fma(-h[0], w[1], fma(-h[1], w[2], y[0]));
}
__device__ __forceinline__ double dot3(const double (&a)[3], const double (&b)[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}

// Z H Z^T (packed) from Z and the metric's factor, with V and Y = V diag(e)
__device__ __forceinline__ void left_metric(const double (&Z)[3][3], const double (&h)[6], double (&V)[3][3],
                                            double (&Y)[3][3], double (&b)[6]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    row_v(Z[c], h, V[c]);
    row_e(V[c], h, Y[c]);
  }
  b[0] = dot3(Y[0], V[0]);
  b[1] = dot3(Y[1], V[1]);
  b[2] = dot3(Y[2], V[2]);
  b[3] = dot3(Y[0], V[1]);
  b[4] = dot3(Y[0], V[2]);
  b[5] = dot3(Y[1], V[2]);
}

// scale * (dev((t1 B^2 + t2 B) / J) + p I) from b = Z H Z^T (packed) and J
__device__ __forceinline__ void stress(const double (&b)[6], double J, double p, double c1, double c2, double scale,
                                       double (&sg)[6]) {
  const double r = rcbrt(J), r2 = r * r, f = r2 * r * scale;  // r^3 = 1 / J
  double B[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) B[i] = r2 * b[i];
  const double I1 = B[0] + B[1] + B[2];
  const double a1 = -2.0 * c2 * f, a2 = 2.0 * fma(I1, c2, c1) * f;
  double S[6];  // a1 B + a2 I
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    S[i] = fma(a1, B[i], a2);
    S[i + 3] = a1 * B[i + 3];
  }
  sg[0] = B[0] * S[0] + B[3] * S[3] + B[4] * S[4];
  sg[1] = B[3] * S[3] + B[1] * S[1] + B[5] * S[5];
  sg[2] = B[4] * S[4] + B[5] * S[5] + B[2] * S[2];
  sg[3] = B[0] * S[3] + B[3] * S[1] + B[4] * S[5];
  sg[4] = B[0] * S[4] + B[3] * S[5] + B[4] * S[2];
  sg[5] = B[3] * S[4] + B[1] * S[5] + B[5] * S[2];
  const double h = fma(-1.0 / 3.0, sg[0] + sg[1] + sg[2], p * scale);
  sg[0] += h;
  sg[1] += h;
  sg[2] += h;
}

}  // namespace mr_sf
