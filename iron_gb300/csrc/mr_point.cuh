// mr_point.cuh -- Gauss-point formulas shared by the Mooney-Rivlin kernels: Voigt maps, Iron's
// cofactor inverse, volume Jacobians, kinematics and Iron's analytic tangent tensors.
#pragma once

#include "df.cuh"
#include "gfe_internal.cuh"

namespace {

constexpr int NQ = 27;   // quadratic element nodes
constexpr int NL = 8;    // linear (pressure) element nodes
constexpr int NG = 27;   // Gauss points (3x3x3)
constexpr int ND = 89;   // element DOFs

// Voigt index of tensor entry (i, j) and the tensor entries of Voigt index v, as arithmetic so that
// unrolled loops index register arrays with constants: 11 22 33 12 13 23.
__host__ __device__ constexpr int t2v(int i, int j) { return i == j ? i : i + j + 2; }
__host__ __device__ constexpr int v2t_a(int v) { return v < 3 ? v : (v == 5 ? 1 : 0); }
__host__ __device__ constexpr int v2t_b(int v) { return v < 3 ? v : (v == 3 ? 1 : 2); }

// Inverse and determinant with Iron's cofactor formulas (src/maths.F90:2807-2868).
template <typename S>
__device__ __forceinline__ S inv3(const S A[3][3], S B[3][3]) {
  const S det = A[0][0] * A[1][1] * A[2][2] + A[0][1] * A[1][2] * A[2][0] + A[0][2] * A[1][0] * A[2][1] -
                A[0][0] * A[2][1] * A[1][2] - A[1][0] * A[0][1] * A[2][2] - A[2][0] * A[1][1] * A[0][2];
  const S r = S(1) / det;
  B[0][0] = (A[1][1] * A[2][2] - A[2][1] * A[1][2]) * r;
  B[1][0] = (A[1][2] * A[2][0] - A[2][2] * A[1][0]) * r;
  B[2][0] = (A[1][0] * A[2][1] - A[2][0] * A[1][1]) * r;
  B[0][1] = (A[2][1] * A[0][2] - A[0][1] * A[2][2]) * r;
  B[1][1] = (A[2][2] * A[0][0] - A[0][2] * A[2][0]) * r;
  B[2][1] = (A[2][0] * A[0][1] - A[0][0] * A[2][1]) * r;
  B[0][2] = (A[0][1] * A[1][2] - A[1][1] * A[0][2]) * r;
  B[1][2] = (A[0][2] * A[1][0] - A[1][2] * A[0][0]) * r;
  B[2][2] = (A[0][0] * A[1][1] - A[1][0] * A[0][1]) * r;
  return det;
}

template <typename S>
__device__ __forceinline__ S det3(const S A[3][3]) {
  return A[0][0] * A[1][1] * A[2][2] + A[0][1] * A[1][2] * A[2][0] + A[0][2] * A[1][0] * A[2][1] -
         A[0][0] * A[2][1] * A[1][2] - A[1][0] * A[0][1] * A[2][2] - A[2][0] * A[1][1] * A[0][2];
}

// Volume Jacobian sqrt|det(M^T M)| (src/coordinate_routines.F90:818-822).
__device__ __forceinline__ double vol_jacobian(const double M[3][3]) {
  double G[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) G[i][j] = M[0][i] * M[0][j] + M[1][i] * M[1][j] + M[2][i] * M[2][j];
  return sqrt(fabs(det3(G)));
}
// The FP32 path keeps the volume Jacobian in FP64: the gradient matrix is widened exactly (integer
// re-packing, no FP64-pipe conversion) and |det M| (= sqrt(det(M^T M)) for a square M) is taken
// directly, which also avoids the Gram product and the square root.
__device__ __forceinline__ float vol_jacobian(const float M[3][3]) {
  double D[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) D[i][j] = f32_to_f64_exact(M[i][j]);
  return (float)fabs(det3(D));
}

// Per-Gauss-point kinematics shared by residual and Jacobian.
template <typename S>
struct GPT {
  S Zi[3][3];  // dxi/dz
  S F[3][3];   // dz/dnu
  S Jz, Jx, p, w;
};
using GP = GPT<double>;

// Jacobians, Z^-1 and the deformation gradient in Iron's fibre-free material frame from Z and X;
// returns det(Z).
template <typename S>
__device__ __forceinline__ S point_frame(const S (&Z)[3][3], const S (&X)[3][3], GPT<S>& o) {
  o.Jz = vol_jacobian(Z);
  o.Jx = vol_jacobian(X);
  const S dz = inv3(Z, o.Zi);
  // material frame without fibres: dX/dNu columns = normalised DX_DXI columns
  S N[3][3], NX[3][3], A[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const S n = sqrt(X[0][k] * X[0][k] + X[1][k] * X[1][k] + X[2][k] * X[2][k]);
#pragma unroll
    for (int c = 0; c < 3; ++c) N[c][k] = X[c][k] / n;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) NX[i][j] = N[0][i] * X[0][j] + N[1][i] * X[1][j] + N[2][i] * X[2][j];
  inv3(NX, A);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) o.F[i][j] = Z[i][0] * A[0][j] + Z[i][1] * A[1][j] + Z[i][2] * A[2][j];
  return dz;
}

// push-forward matrix t (src/finite_elasticity_routines.F90:1343-1375)
template <typename S>
__device__ __forceinline__ void push_t(const S F[3][3], S t[6][6]) {
#pragma unroll
  for (int j = 0; j < 6; ++j)
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int ai = v2t_a(i), bi = v2t_b(i), aj = v2t_a(j), bj = v2t_b(j);
      S v = F[ai][aj] * F[bi][bj];
      if (j >= 3) v += F[ai][bj] * F[bi][aj];
      t[i][j] = v;
    }
}

template <typename R>
__device__ __forceinline__ void push_vec(const R t[6][6], R S[6], R J) {
  R o[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    R s = R(0);
#pragma unroll
    for (int j = 0; j < 6; ++j) s += t[i][j] * S[j];
    o[i] = s / J;
  }
#pragma unroll
  for (int i = 0; i < 6; ++i) S[i] = o[i];
}

// Iron's per-Gauss-point tangent blocks in spatial coordinates (src/finite_elasticity_routines.F90:
// 649-795 and 1072-1192): sub[0..2] = J_z w (c_sub + sigma) for the diagonal component blocks,
// sub[3..5] = J_z w c_sub for the off-diagonal blocks (mh, nh) = (1,0), (2,0), (2,1);
// hyd = J_z w push(C^-1).
template <typename S>
__device__ void iron_point_tensors(const GPT<S>& q, S c1, S c2, S sub[6][9], S hyd[9], S& jgw) {
  const S J = q.Jz / q.Jx;
  // unmodified right Cauchy-Green tensor and its inverse
  S C[3][3], Ci[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) C[i][j] = q.F[0][i] * q.F[0][j] + q.F[1][i] * q.F[1][j] + q.F[2][i] * q.F[2][j];
  const S I3 = inv3(C, Ci);
  const S L[6] = {C[0][0], C[1][1], C[2][2], C[0][1], C[0][2], C[1][2]};
  const S U[6] = {Ci[0][0], Ci[1][1], Ci[2][2], Ci[0][1], Ci[0][2], Ci[1][2]};
  // I3EE as filled by Fortran RESHAPE (column j listed): I3EE[i][j] = col[j][i]
  const S z0 = S(0), f4 = S(4), f2 = S(2);
  const S col[6][6] = {{z0, f4 * L[2], f4 * L[1], z0, z0, -f4 * L[5]},
                       {f4 * L[2], z0, f4 * L[0], z0, -f4 * L[4], z0},
                       {f4 * L[1], f4 * L[0], z0, -f2 * L[3], z0, z0},
                       {z0, z0, -f4 * L[3], -f2 * L[2], f2 * L[5], f2 * L[4]},
                       {z0, -f4 * L[4], z0, f2 * L[5], -f2 * L[1], f2 * L[3]},
                       {-f4 * L[5], z0, z0, f2 * L[4], f2 * L[3], -f2 * L[0]}};
  S D[6][6];
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      S v = S(0);
      if (i < 3 && j < 3 && i != j) v = f4 * c2;
      if (i >= 3 && i == j) v = -f2 * c2;
      D[i][j] = v + q.p * (-f2 * U[i] * U[j] + S(0.5) * col[j][i] / I3);
    }
  const S I1 = C[0][0] + C[1][1] + C[2][2];
  const S t2 = f2 * (c1 + I1 * c2);
  S Sv[6] = {-f2 * c2 * C[0][0] + t2, -f2 * c2 * C[1][1] + t2, -f2 * c2 * C[2][2] + t2,
             -f2 * c2 * C[1][0], -f2 * c2 * C[2][0], -f2 * c2 * C[2][1]};
  S H[6] = {U[0], U[1], U[2], U[3], U[4], U[5]};
  S t[6][6];
  push_t(q.F, t);
  push_vec(t, Sv, J);
  push_vec(t, H, J);
  S tD[6][6];
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      S s = S(0);
#pragma unroll
      for (int k = 0; k < 6; ++k) s += t[i][k] * D[k][j];
      tD[i][j] = s;
    }
#pragma unroll
  for (int i = 0; i < 6; ++i)
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      S s = S(0);
#pragma unroll
      for (int k = 0; k < 6; ++k) s += tD[i][k] * t[j][k];
      D[i][j] = s / J;
    }
  Sv[0] += q.p; Sv[1] += q.p; Sv[2] += q.p;
  jgw = q.Jz * q.w;
#pragma unroll
  for (int nh = 0; nh < 3; ++nh)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) sub[nh][i * 3 + j] = jgw * (D[t2v(i, nh)][t2v(j, nh)] + Sv[t2v(i, j)]);
  const int om[3] = {1, 2, 2}, on[3] = {0, 0, 1};
#pragma unroll
  for (int o = 0; o < 3; ++o)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) sub[3 + o][i * 3 + j] = jgw * D[t2v(i, om[o])][t2v(j, on[o])];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) hyd[i * 3 + j] = jgw * H[t2v(i, j)];
}

}  // namespace
