// mr_jac64.cu -- FP64 element Jacobians of the Q2/Q1 Mooney-Rivlin element, sum-factorised.
//
// Both kernels are bound by GB300's FP64 pipe (one warp instruction in 64 cycles), so their design
// is about issuing fewer FP64 instructions on full warps.
//
// K(ms mh, ns nh) = sum_g g_ms^T D_g^(mh,nh) g_ns with the reference basis gradients g and 3x3 blocks
// D_g[xi][zeta] at 27 Gauss points, and the u-p / p-u blocks from Hv_g[xi][mh], Pv_g[xi][nh]:
//  * mr_point_blocks64, one thread per (element, point), eight elements a CTA: the gradients by
//    mr_sf.cuh, then the blocks in closed form (consistent tangent) or Iron's tensors.  The consistent
//    tangent took ten forward-mode dual passes a point, about 9,000 operations; the closed form of
//    dP/dZ below takes about 550.
//  * mr_contract64, one CTA per element: the contraction one xi direction at a time over pairs of 1D
//    functions (test a, trial b).  A line of three point values gives its nine pair sums in 11 to 20
//    operations (the point 1/2 only meets one or two functions, the outer points share products).  The
//    nine (xi, zeta) terms merge into the four kinds that differ in the third direction before it.
//    About 75,000 operations an element; the dense product 243 x 81 by 81 x 27 with its operand and
//    the dense u-p sums took 690,000.
// Only the six blocks mh >= nh are formed: Iron mirrors its lower triangle, and the consistent
// tangent is symmetric.
// Measured at 15 x 18 x 13 elements, point + contraction kernels: 1.87 + 4.23 ms before, 0.14 + 0.64 ms here.
#include <algorithm>

#include "mr_jac64.cuh"
#include "mr_point.cuh"
#include "mr_sf.cuh"

namespace {

constexpr int kPointElems = 8;                    // elements a CTA of the point kernel
constexpr int kPointThreads = kPointElems * NG;   // 216: 27 points an element on 6.75 warps
constexpr int kChunk = 1 << 16;                   // elements whose point blocks are held at a time

// point blocks of one element: 54 rows D (blocks (0,0) (1,1) (2,2) (1,0) (2,0) (2,1), each [xi][zeta]),
// 9 rows Hv[xi][mh], and for Iron's Jacobian 9 rows Pv[xi][nh] (equal to Hv in the consistent tangent);
// a row holds the 27 points, so the point kernel's stores and the contraction's lines are contiguous
template <bool EXACT>
constexpr int kBlockRows = EXACT ? 63 : 72;

struct PointShared {
  double u[2][81], A[162], B[243], grad[243], p[NL];
};

// dP/dZ of the consistent tangent at one point in closed form.  With sigma_bar = S = a1 B^2 + a2 B
// (a1 = -2 c2 / J, a2 = 2 (c1 + I1 c2) / J, B = J^(-2/3) Z H Z^T, mr_sf.cuh) and a velocity gradient l
// (dZ = l Z), d(J sigma) and d(Z^-1) give P's derivative as J_z w Z^-1 a Z^-T with
//   a_{imnj} = delta_mn S_ij + k1 delta_in delta_jm + (a1)(B_ij B_mn + B_in B_jm) - 2 a1 B_im B_nj
//              - delta_nj Q_im - delta_im Q_nj + k2 delta_im delta_nj,
//   Q = 4/3 a1 B^2 + (4/3 c2 I1 / J + 2/3 a2) B,  k1 = tr(S)/3 - p,  k2 = tr(Q)/3 + p
// (4 c2 / J = -2 a1).  Pulled back with the cofactor rows z_m of Z (Z^-1 = z / det): w / |det Z| times
//   D^(mn) = B_mn a1 BB + delta_mn SS + k1 z_n z_m^T + a1 (Bz_n Bz_m^T - 2 Bz_m Bz_n^T)
//            - Y_m z_n^T - z_m Y_n^T,  Y_m = Qz_m - k2/2 z_m,
// Bz_m = sum_i B_im z_i, BB = sum_i z_i Bz_i^T, SS = sum_ij S_ij z_i z_j^T.
__device__ __forceinline__ void exact_blocks(const double (&Z)[3][3], const double (&X)[3][3], double p, double w,
                                             double c1, double c2, double* __restrict__ o, unsigned* err) {
  double h[6], z[3][3], B[6];
  const double Jx = mr_sf::geometry(X, h);
  const double det = mr_sf::cofactors(Z, z);
  if (!(det > 0.0) || !isfinite(det)) gfe_raise(err, GFE_DEVERR_JACOBIAN);
  const double J = fabs(det) / Jx;
  const double r = rcbrt(J), r2 = r * r, iJ = r2 * r;
  {
    double V[3][3], Y[3][3];
    mr_sf::left_metric(Z, h, V, Y, B);
#pragma unroll
    for (int i = 0; i < 6; ++i) B[i] *= r2;
  }
  const double I1 = B[0] + B[1] + B[2];
  const double a1 = -2.0 * c2 * iJ, a2 = 2.0 * fma(I1, c2, c1) * iJ;
  // Hv = dP/dp = w J_z Z^-1 (before z is scaled)
  const double ws = det > 0.0 ? w : -w;
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) o[(54 + k * 3 + c) * NG] = ws * z[c][k];
  // z scaled by sqrt(w / |det|) once: every term is quadratic in z
  const double f = sqrt(w / fabs(det));
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) z[c][k] *= f;
  const double trB2 = B[0] * B[0] + B[1] * B[1] + B[2] * B[2] + 2.0 * (B[3] * B[3] + B[4] * B[4] + B[5] * B[5]);
  const double beta = fma(4.0 / 3.0 * c2 * iJ, I1, 2.0 / 3.0 * a2), q1 = 4.0 / 3.0 * a1;
  const double k1 = fma(a1, trB2, a2 * I1) * (1.0 / 3.0) - p;
  const double k2h = 0.5 * (fma(q1, trB2, beta * I1) * (1.0 / 3.0) + p);
  double Bz[3][3], Y[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Bz[0][k] = B[0] * z[0][k] + B[3] * z[1][k] + B[4] * z[2][k];
    Bz[1][k] = B[3] * z[0][k] + B[1] * z[1][k] + B[5] * z[2][k];
    Bz[2][k] = B[4] * z[0][k] + B[5] * z[1][k] + B[2] * z[2][k];
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double s0 = B[0] * Bz[0][k] + B[3] * Bz[1][k] + B[4] * Bz[2][k];
    const double s1 = B[3] * Bz[0][k] + B[1] * Bz[1][k] + B[5] * Bz[2][k];
    const double s2 = B[4] * Bz[0][k] + B[5] * Bz[1][k] + B[2] * Bz[2][k];
    Y[0][k] = fma(q1, s0, fma(beta, Bz[0][k], -k2h * z[0][k]));
    Y[1][k] = fma(q1, s1, fma(beta, Bz[1][k], -k2h * z[1][k]));
    Y[2][k] = fma(q1, s2, fma(beta, Bz[2][k], -k2h * z[2][k]));
  }
  double T1[3][3], T2[3][3];  // a1 BB and SS
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) {
      const double bb = z[0][i] * Bz[0][j] + z[1][i] * Bz[1][j] + z[2][i] * Bz[2][j];
      const double b2 = Bz[0][i] * Bz[0][j] + Bz[1][i] * Bz[1][j] + Bz[2][i] * Bz[2][j];
      T1[i][j] = T1[j][i] = a1 * bb;
      T2[i][j] = T2[j][i] = fma(a1, b2, a2 * bb);
    }
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {
        double v = fma(B[m], T1[i][j], T2[i][j]);
        v = fma(k1 * z[m][i], z[m][j], v);
        v = fma(-a1 * Bz[m][i], Bz[m][j], v);
        v = fma(-Y[m][i], z[m][j], v);
        v = fma(-z[m][i], Y[m][j], v);
        o[(m * 9 + i * 3 + j) * NG] = v;
        if (i != j) o[(m * 9 + j * 3 + i) * NG] = v;
      }
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int m = q == 0 ? 1 : 2, n = q == 2 ? 1 : 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double zk = k1 * z[n][i], bn = a1 * Bz[n][i], bm = -2.0 * a1 * Bz[m][i];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        double v = B[3 + q] * T1[i][j];
        v = fma(zk, z[m][j], v);
        v = fma(bn, Bz[m][j], v);
        v = fma(bm, Bz[n][j], v);
        v = fma(-Y[m][i], z[n][j], v);
        v = fma(-z[m][i], Y[n][j], v);
        o[((3 + q) * 9 + i * 3 + j) * NG] = v;
      }
    }
  }
}

// Iron's analytic tangent: the spatial blocks of iron_point_tensors mapped to xi space.
__device__ __forceinline__ void iron_blocks(const double (&Z)[3][3], const double (&X)[3][3], double p, double w,
                                            double c1, double c2, double* __restrict__ o, unsigned* err) {
  GP q;
  const double dz = point_frame(Z, X, q);
  q.p = p;
  q.w = w;
  if (!(dz > 0.0 && q.Jx > 0.0 && isfinite(dz))) gfe_raise(err, GFE_DEVERR_JACOBIAN);
  double sub[6][9], hyd[9], jgw;
  iron_point_tensors(q, c1, c2, sub, hyd, jgw);
#pragma unroll
  for (int blk = 0; blk < 6; ++blk) {
    double W[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int z = 0; z < 3; ++z)
        W[i][z] = sub[blk][i * 3] * q.Zi[z][0] + sub[blk][i * 3 + 1] * q.Zi[z][1] + sub[blk][i * 3 + 2] * q.Zi[z][2];
#pragma unroll
    for (int xi = 0; xi < 3; ++xi)
#pragma unroll
      for (int z = 0; z < 3; ++z)
        o[(blk * 9 + xi * 3 + z) * NG] = q.Zi[xi][0] * W[0][z] + q.Zi[xi][1] * W[1][z] + q.Zi[xi][2] * W[2][z];
  }
#pragma unroll
  for (int xi = 0; xi < 3; ++xi)
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      o[(54 + xi * 3 + m) * NG] = q.Zi[xi][0] * hyd[m * 3] + q.Zi[xi][1] * hyd[m * 3 + 1] + q.Zi[xi][2] * hyd[m * 3 + 2];
      o[(63 + xi * 3 + m) * NG] = jgw * q.Zi[xi][m];
    }
}

template <bool EXACT>
__global__ void __launch_bounds__(kPointThreads, EXACT ? 2 : 1)  // Iron's 6x6 tensors need 255 registers
mr_point_blocks64(const int32_t* __restrict__ elems, int32_t count, const int32_t* __restrict__ eq2,
                  const int32_t* __restrict__ elin, int32_t nq2, const double* __restrict__ xg,
                  const double* __restrict__ dep, const double* __restrict__ cpar, double* __restrict__ out,
                  unsigned* err) {
  extern __shared__ double smem[];
  const int le = threadIdx.x / NG, g = threadIdx.x % NG;
  PointShared& S = reinterpret_cast<PointShared*>(smem)[le];
  const int item = blockIdx.x * kPointElems + le;
  const bool on = item < count;
  if (on) {
    const int e = __ldg(elems + item);
    const int n = __ldg(eq2 + (size_t)e * NQ + g);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      S.u[0][c * NQ + g] = __ldg(xg + (size_t)c * nq2 + n);
      S.u[1][c * NQ + g] = dep[(size_t)c * nq2 + n];
    }
    if (g < NL) S.p[g] = dep[(size_t)3 * nq2 + __ldg(elin + (size_t)e * NL + g)];
  }
  auto sync = [] { __syncthreads(); };
  double X[3][3], Z[3][3];
  sync();
  mr_sf::field_gradients(g, on, S.u[0], S.A, S.B, S.grad, sync);
  sync();
#pragma unroll
  for (int i = 0; i < 9; ++i) X[i / 3][i % 3] = S.grad[i * NG + g];
  mr_sf::field_gradients(g, on, S.u[1], S.A, S.B, S.grad, sync);
  sync();
  if (!on) return;
#pragma unroll
  for (int i = 0; i < 9; ++i) Z[i / 3][i % 3] = S.grad[i * NG + g];
  const double p = mr_sf::point_pressure(g, S.p), w = mr_sf::point_weight(g);
  double* o = out + (size_t)item * (kBlockRows<EXACT> * NG) + g;
  if constexpr (EXACT) exact_blocks(Z, X, p, w, cpar[0], cpar[1], o, err);
  else iron_blocks(Z, X, p, w, cpar[0], cpar[1], o, err);
}

// ---- contraction ----------------------------------------------------------------------------------
// Products of the 1D functions at the Gauss points 1/2 - t, 1/2, 1/2 + t: values (va, .4, vb), (0, 1, 0),
// (vb, .4, va) and slopes (-dp, dq, -dm), (-1, 0, 1), (dm, -dq, dp).
constexpr double kVa = 0.3 + mr_sf::kT, kVb = 0.3 - mr_sf::kT, kVm = 0.4;
constexpr double kDp = mr_sf::k4T + 1.0, kDm = mr_sf::k4T - 1.0, kDq = mr_sf::k8T;

template <bool ADD>
__device__ __forceinline__ void put2(double& o, double c0, double s0, double c2, double s2) {
  o = ADD ? fma(c0, s0, fma(c2, s2, o)) : fma(c0, s0, c2 * s2);
}

// o[a * 3 + b] (+)= sum_g f_a(g) h_b(g) s_g, f / h the values or slopes of test / trial function
template <bool FD, bool HD, bool ADD>
__device__ __forceinline__ void pair_line(double s0, double s1, double s2, double (&o)[9]) {
  if constexpr (!FD && !HD) {
    const double s = s0 + s2;
    const double u = fma(kVa * kVm, s0, kVb * kVm * s2), v = fma(kVb * kVm, s0, kVa * kVm * s2);
    put2<ADD>(o[0], kVa * kVa, s0, kVb * kVb, s2);
    put2<ADD>(o[8], kVb * kVb, s0, kVa * kVa, s2);
    if constexpr (ADD) {
      o[1] += u; o[3] += u; o[5] += v; o[7] += v;
      o[2] = fma(kVa * kVb, s, o[2]);
      o[6] = fma(kVa * kVb, s, o[6]);
      o[4] += fma(kVm * kVm, s, s1);
    } else {
      o[1] = o[3] = u;
      o[5] = o[7] = v;
      o[2] = o[6] = kVa * kVb * s;
      o[4] = fma(kVm * kVm, s, s1);
    }
  } else if constexpr (FD && HD) {
    const double s = s0 + s2;
    const double u = fma(-kDp * kDq, s0, -kDm * kDq * s2), v = fma(-kDq * kDm, s0, -kDq * kDp * s2);
    const double d = fma(kDp * kDm, s, -s1);
    if constexpr (ADD) {
      o[0] += fma(kDp * kDp, s0, fma(kDm * kDm, s2, s1));
      o[8] += fma(kDm * kDm, s0, fma(kDp * kDp, s2, s1));
      o[1] += u; o[3] += u; o[5] += v; o[7] += v;
      o[2] += d; o[6] += d;
      o[4] = fma(kDq * kDq, s, o[4]);
    } else {
      o[0] = fma(kDp * kDp, s0, fma(kDm * kDm, s2, s1));
      o[8] = fma(kDm * kDm, s0, fma(kDp * kDp, s2, s1));
      o[1] = o[3] = u;
      o[5] = o[7] = v;
      o[2] = o[6] = d;
      o[4] = kDq * kDq * s;
    }
  } else {
    // value function index i, slope function index j at o[i * si + j * sj]
    constexpr int si = FD ? 1 : 3, sj = FD ? 3 : 1;
    put2<ADD>(o[0], -kVa * kDp, s0, kVb * kDm, s2);
    put2<ADD>(o[sj], kVa * kDq, s0, -kVb * kDq, s2);
    put2<ADD>(o[2 * sj], -kVa * kDm, s0, kVb * kDp, s2);
    put2<ADD>(o[2 * si], -kVb * kDp, s0, kVa * kDm, s2);
    put2<ADD>(o[2 * si + sj], kVb * kDq, s0, -kVa * kDq, s2);
    put2<ADD>(o[2 * si + 2 * sj], -kVb * kDm, s0, kVa * kDp, s2);
    put2<ADD>(o[si + sj], kVm * kDq, s0, -kVm * kDq, s2);
    if constexpr (ADD) {
      o[si] += fma(-kVm * kDp, s0, fma(kVm * kDm, s2, -s1));
      o[si + 2 * sj] += fma(-kVm * kDm, s0, fma(kVm * kDp, s2, s1));
    } else {
      o[si] = fma(-kVm * kDp, s0, fma(kVm * kDm, s2, -s1));
      o[si + 2 * sj] = fma(-kVm * kDm, s0, fma(kVm * kDp, s2, s1));
    }
  }
}

// o[a * 2 + b] (+)= sum_g f_a(g) l_b(g) s_g with the linear functions l_0 = 1 - x, l_1 = x
template <bool FD, bool ADD>
__device__ __forceinline__ void up_line(double s0, double s1, double s2, double (&o)[6]) {
  double t[3], u[3];
  const double x0 = (0.5 - mr_sf::kT) * s0, x1 = 0.5 * s1, x2 = (0.5 + mr_sf::kT) * s2;
  if constexpr (FD) {
    mr_sf::line_der_t(s0, s1, s2, t);
    mr_sf::line_der_t(x0, x1, x2, u);
  } else {
    mr_sf::line_val_t(s0, s1, s2, t);
    mr_sf::line_val_t(x0, x1, x2, u);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if constexpr (ADD) {
      o[a * 2] += t[a] - u[a];
      o[a * 2 + 1] += u[a];
    } else {
      o[a * 2] = t[a] - u[a];
      o[a * 2 + 1] = u[a];
    }
  }
}

constexpr int kC64Threads = 256;  // two CTAs an SM (98 KB of shared memory, 128 registers)

// second[] first holds the element's point blocks; first[] is reused for the finished blocks
template <bool EXACT>
struct Contract64 {
  static constexpr int kSets = EXACT ? 1 : 2;  // u-p, and p-u where it differs
  double first[6 * 729 + kSets * 648];   // [blk][type][pair1][line], then u-p [set][mh][xi][pair1 (6)][line]
  double second[6 * 972 + kSets * 648];  // [blk][kind][pair2][pair1][g3], then [set][mh][kind][pair2][pair1][g3]
};

template <bool EXACT>
__global__ void __launch_bounds__(kC64Threads, 2)
mr_contract64(const int32_t* __restrict__ elems, int32_t count, const double* __restrict__ gp,
              double* __restrict__ Kel) {
  extern __shared__ double smem[];
  using Sh = Contract64<EXACT>;
  Sh& S = *reinterpret_cast<Sh*>(smem);
  constexpr int kIn = kBlockRows<EXACT> * NG;
  static_assert(kIn <= 6 * 972, "the point blocks fit in the second stage's array");
  const int tid = threadIdx.x;
  double* up1 = S.first + 6 * 729;
  double* up2 = S.second + 6 * 972;
  for (int item = blockIdx.x; item < count; item += gridDim.x) {
    // (the previous element's last reads of second[] lie before a barrier)
    const double* src = gp + (size_t)item * kIn;
    for (int t = tid; t < kIn; t += kC64Threads) S.second[t] = __ldcs(src + t);
    __syncthreads();
    // xi1: unit (type, blk, line), the types ordered by the functions they take in xi1 (slope-slope,
    // slope-value, value-slope, value-value) so that few warps mix two of them
    for (int u = tid; u < 486 + Sh::kSets * 81; u += kC64Threads) {
      if (u < 486) {
        const int ty = u / 54, blk = (u % 54) / 9, line = u % 9;
        const int type = ty == 0 ? 0 : (ty < 3 ? ty : (ty == 3 ? 3 : (ty == 4 ? 6 : ty + (ty >= 7 ? 0 : -1))));
        const double* s = S.second + (blk * 9 + type) * NG + line * 3;
        double o[9];
        if (ty == 0) pair_line<true, true, false>(s[0], s[1], s[2], o);
        else if (ty < 3) pair_line<true, false, false>(s[0], s[1], s[2], o);
        else if (ty < 5) pair_line<false, true, false>(s[0], s[1], s[2], o);
        else pair_line<false, false, false>(s[0], s[1], s[2], o);
        double* d = S.first + (blk * 9 + type) * 81 + line;
#pragma unroll
        for (int q = 0; q < 9; ++q) d[q * 9] = o[q];
      } else {
        const int v = u - 486, xi = v / (27 * Sh::kSets), r = v % (27 * Sh::kSets);
        const int set = r / 27, mh = (r % 27) / 9, line = r % 9;
        const double* s = S.second + (54 + set * 9 + xi * 3 + mh) * NG + line * 3;
        double o[6];
        if (xi == 0) up_line<true, false>(s[0], s[1], s[2], o);
        else up_line<false, false>(s[0], s[1], s[2], o);
        double* d = up1 + ((set * 3 + mh) * 3 + xi) * 54 + line;
#pragma unroll
        for (int q = 0; q < 6; ++q) d[q * 9] = o[q];
      }
    }
    __syncthreads();
    // xi2: unit (blk, pair1, g3); the four kinds by the functions taken in xi3: 0 value-value (four
    // types), 1 slope-value, 2 value-slope, 3 slope-slope; one group of units takes kind 0, one the rest
    for (int u = tid; u < 324 + Sh::kSets * 54; u += kC64Threads) {
      if (u < 324) {
        const int v = u % 162, blk = v / 27, m = v % 27;
        const double* s = S.first + blk * 729 + m * 3;
        double* d = S.second + blk * 972 + m;
        double o[9];
        auto at = [&](int type, int g) { return s[type * 81 + g]; };
        auto store = [&](int kind) {
#pragma unroll
          for (int q = 0; q < 9; ++q) d[(kind * 9 + q) * 27] = o[q];
        };
        if (u < 162) {
          pair_line<false, false, false>(at(0, 0), at(0, 1), at(0, 2), o);
          pair_line<false, true, true>(at(1, 0), at(1, 1), at(1, 2), o);
          pair_line<true, false, true>(at(3, 0), at(3, 1), at(3, 2), o);
          pair_line<true, true, true>(at(4, 0), at(4, 1), at(4, 2), o);
          store(0);
        } else {
          pair_line<false, false, false>(at(6, 0), at(6, 1), at(6, 2), o);
          pair_line<false, true, true>(at(7, 0), at(7, 1), at(7, 2), o);
          store(1);
          pair_line<false, false, false>(at(2, 0), at(2, 1), at(2, 2), o);
          pair_line<true, false, true>(at(5, 0), at(5, 1), at(5, 2), o);
          store(2);
          pair_line<false, false, false>(at(8, 0), at(8, 1), at(8, 2), o);
          store(3);
        }
      } else {
        const int v = u - 324, f = v / 18, m = v % 18;  // f = set * 3 + mh, m = pair1 * 3 + g3
        const double* s = up1 + f * 162 + m * 3;
        double* d = up2 + f * 216 + m;
        double o[6];
        up_line<false, false>(s[0], s[1], s[2], o);
        up_line<true, true>(s[54], s[55], s[56], o);
#pragma unroll
        for (int q = 0; q < 6; ++q) d[q * 18] = o[q];
        up_line<false, false>(s[108], s[109], s[110], o);
#pragma unroll
        for (int q = 0; q < 6; ++q) d[(6 + q) * 18] = o[q];
      }
    }
    __syncthreads();
    // xi3: unit (blk, pair2, pair1); pair (a, b) of function indices, ms = a1 + 3 a2 + 9 a3
    for (int u = tid; u < 486 + Sh::kSets * 108; u += kC64Threads) {
      if (u < 486) {
        const int blk = u / 81, pair2 = (u % 81) / 9, pair1 = u % 9;
        const double* s = S.second + blk * 972 + pair2 * 27 + pair1 * 3;
        double o[9];
        pair_line<false, false, false>(s[0], s[1], s[2], o);
        pair_line<true, false, true>(s[243], s[244], s[245], o);
        pair_line<false, true, true>(s[486], s[487], s[488], o);
        pair_line<true, true, true>(s[729], s[730], s[731], o);
        double* d = S.first + blk * 729 + (pair1 / 3 + 3 * (pair2 / 3)) * 27 + pair1 % 3 + 3 * (pair2 % 3);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 3; ++b) d[a * 243 + b * 9] = o[a * 3 + b];
      } else {
        const int v = u - 486, f = v / 36, pair2 = (v % 36) / 6, pair1 = v % 6;
        const double* s = up2 + f * 216 + pair2 * 18 + pair1 * 3;
        double o[6];
        up_line<false, false>(s[0], s[1], s[2], o);
        up_line<true, true>(s[108], s[109], s[110], o);
        // up1[set][mh][ms][b], b = b1 + 2 b2 + 4 b3
        double* d = up1 + f * 216 + (pair1 / 2 + 3 * (pair2 / 2)) * 8 + pair1 % 2 + 2 * (pair2 % 2);
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b) d[a * 72 + b * 4] = o[a * 2 + b];
      }
    }
    __syncthreads();
    // the element matrix, a warp a row: lower blocks as formed, the upper triangle mirrored
    double* Ke = Kel + (size_t)__ldg(elems + item) * ND * ND;
    const int lane = tid & 31;
    for (int r = tid >> 5; r < ND; r += kC64Threads / 32) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int c = lane + 32 * j;
        if (c >= ND) continue;
        double v = 0.0;
        if (r < 81 && c < 81) {
          const int hi = r >= c ? r : c, lo = r >= c ? c : r;
          const int mh = hi / 27, nh = lo / 27;
          const int blk = mh == nh ? mh : (mh == 1 ? 3 : 4 + nh);
          v = S.first[blk * 729 + (hi - 27 * mh) * 27 + lo - 27 * nh];
        } else if (r < 81) {
          v = up1[r * 8 + c - 81];
        } else if (c < 81) {
          v = up1[(Sh::kSets - 1) * 648 + c * 8 + r - 81];
        }
        __stcs(Ke + (size_t)r * ND + c, v);
      }
    }
    // first[] is rewritten after the barrier that follows the next element's load
  }
}

}  // namespace

namespace mr64 {

template <bool EXACT>
static int run(int32_t n_elem, const int32_t* elems, const int32_t* eq2, const int32_t* elin, int32_t nq2,
               const double* xg, const double* dep, const double* cpar, double* Kel, cudaStream_t s, unsigned* err,
               int* launches) {
  const size_t psm = sizeof(PointShared) * kPointElems, csm = sizeof(Contract64<EXACT>);
  GFE_CUDA_TRY(cudaFuncSetAttribute((const void*)mr_point_blocks64<EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)psm));
  GFE_CUDA_TRY(cudaFuncSetAttribute((const void*)mr_contract64<EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)csm));
  const int chunk = std::min(n_elem, kChunk);
  double* gp = nullptr;
  if (int rc = gfe::scratch_alloc((void**)&gp, sizeof(double) * (size_t)chunk * kBlockRows<EXACT> * NG, s,
                                  "Gauss-point tangent blocks"))
    return rc;
  for (int c0 = 0; c0 < n_elem; c0 += chunk) {
    const int cnt = std::min(chunk, n_elem - c0);
    mr_point_blocks64<EXACT><<<(cnt + kPointElems - 1) / kPointElems, kPointThreads, psm, s>>>(
        elems + c0, cnt, eq2, elin, nq2, xg, dep, cpar, gp, err);
    mr_contract64<EXACT><<<std::min(cnt, 2 * gfe::sm_count()), kC64Threads, csm, s>>>(elems + c0, cnt, gp, Kel);
    *launches += 2;
  }
  gfe::scratch_free(gp, s);
  return GFE_OK;
}

int element_matrices(bool exact, int32_t n_elem, const int32_t* elems, const int32_t* eq2, const int32_t* elin,
                     int32_t nq2, const double* xg, const double* dep, const double* cpar, double* Kel,
                     cudaStream_t s, unsigned* err, int* launches) {
  if (exact) return run<true>(n_elem, elems, eq2, elin, nq2, xg, dep, cpar, Kel, s, err, launches);
  return run<false>(n_elem, elems, eq2, elin, nq2, xg, dep, cpar, Kel, s, err, launches);
}

}  // namespace mr64
