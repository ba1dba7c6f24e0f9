// laplace_tp_sf.cuh -- sum-factorised element matrices of the basis-generic Laplace assembly.
//
// Hexahedra with the same number N of 1D functions in every direction (3: quadratic Lagrange; 4: cubic
// Lagrange and cubic Hermite, also mixed) and N Gauss points a direction, in FP64 and float-float.
// K(m, n) = sum_g dphi_m^T M_g dphi_n is a tensor product: every term is a product over the directions of
// a pair of 1D functions (test a, trial b), each a value V or a slope D:
//   M00 DD VV VV + M11 VV DD VV + M22 VV VV DD            (symmetric in every pair)
//   M01 (DV VD + VD DV) VV,  M02 (DV . VD + ...) VV in 2,  M12 (. DV VD + ...) VV in 1
// so the sums over the Gauss points are taken one direction at a time over pairs:
//   stage 1 (xi1)  X0..X2, X12 over symmetric pairs, X01, X02 over all pairs, for each line
//   stage 2 (xi2)  A = M00 and M11 terms and both M01 terms, for one half of the (a1 a2, b1 b2) pairs (A
//                  is symmetric under their exchange); C = the M22 term; U = the M02 and M12 terms whose
//                  slope in xi3 is the trial function's
//   stage 3 (xi3)  R = A VV + C DD over symmetric pairs, U3 = U VD over all pairs
// and K(m, n) = R + U3(m, n) + U3(n, m).  About 68,000 multiply-adds an element of 64 parameters and 12,500
// of 27; the pairwise sums of laplace_tp_kernel take 1.7 M and 140,000.  The kernel is bound by the FP64
// pipe (FP64) or the FP32 issue rate (float-float); each output of a stage is one thread's unit, so all
// warps work in every stage, and all intermediates stay in shared memory.
// Measured: Hermite FP64, 13 x 11 x 12 elements, 7.71 -> 0.37 ms; Q2 float-float, 36 x 31 x 33, 2.80 ->
// 0.71 ms (pairwise kernel -> this one).
#pragma once

namespace {

template <int N>
struct SFShape {
  static constexpr int Q = N;
  static constexpr int NS = N * (N + 1) / 2, NA = N * N, NH = NA * (NA + 1) / 2;
  static constexpr int NF = N * N * N, NG = Q * Q * Q, NP = NF * (NF + 1) / 2;
  static constexpr int kThreads = N == 3 ? 128 : 256;
  // 1D tables of one direction: values and slopes [function][point], then pair products VV, DD over
  // symmetric pairs and DV (test slope, trial value) over all pairs, [pair][point]
  static constexpr int oD = N * Q, oVV = 2 * N * Q, oDD = oVV + NS * Q, oDV = oDD + NS * Q, kTab = oDV + NA * Q;
  // shared memory, in elements of T; the geometry's arrays lie in U3's place
  static constexpr int sTab = 0, sM = 3 * kTab, sX = sM + 6 * NG, kX = (4 * NS + 2 * NA) * Q * Q;
  static constexpr int sA = sX + kX, sC = sA + NH * Q, sU = sC + NS * NS * Q, sR = sU + NA * NA * Q;
  static constexpr int sU3 = sR + NH * NS, kShared = sU3 + NA * NA * NA;
  static constexpr int gx = sU3, gA = gx + 3 * NF, gB = gA + 6 * N * N * Q, gJ = gB + 9 * N * Q * Q;
  static_assert(gJ + 9 * NG <= kShared, "geometry fits in U3's place");
};

__host__ __device__ constexpr int sym_pair(int a, int b, int n) {  // a <= b
  return a * n - a * (a - 1) / 2 + (b - a);
}
template <int N>
__device__ __forceinline__ int sym_at(int a, int b) {
  return a <= b ? sym_pair(a, b, N) : sym_pair(b, a, N);
}

// one entry pair m <= n of the element matrix: nodes, its place in R, and in U3 both ways round
struct SFPair {
  int32_t mn, r, ab, ba;
};

template <typename T>
struct SFTables {
  T* tab = nullptr;            // three directions
  SFPair* pairs = nullptr;     // [NP]
  int32_t* half = nullptr;     // [NH]: (a1 + N a2) | (b1 + N b2) << 16, first <= second
  int32_t* param = nullptr;    // [NF]: element parameter of the functions (f1, f2, f3), f1 fastest, and
                               // kSFValue unless it is a derivative
};
constexpr int kSFValue = 1 << 16;

__device__ __forceinline__ void mac(double& s, double a, double b) { s = fma(a, b, s); }
__device__ __forceinline__ void mac(f2& s, f2 a, f2 b) { accum(s, a * b); }

// sum_q c[q] * t[q] over n terms, c at stride sc
template <int n, typename T>
__device__ __forceinline__ void dot_add(T& s, const T* c, int sc, const T* t) {
#pragma unroll
  for (int q = 0; q < n; ++q) mac(s, c[q * sc], t[q]);
}

template <typename T, int N>
__global__ void __launch_bounds__(SFShape<N>::kThreads)
laplace_tp_sf_kernel(const int32_t* __restrict__ ce, int32_t cnt, int32_t n_nodes, const int32_t* __restrict__ en,
                     const double* __restrict__ coords, const double* __restrict__ scale,
                     const double* __restrict__ kappa, const T* __restrict__ wg, SFTables<T> tabs,
                     const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const int32_t* __restrict__ slots,
                     double* __restrict__ values, double* __restrict__ Kel, unsigned* err) {
  using Sh = SFShape<N>;
  constexpr int Q = Sh::Q, NS = Sh::NS, NA = Sh::NA, NH = Sh::NH, NF = Sh::NF, NG = Sh::NG, NT = Sh::kThreads;
  extern __shared__ __align__(16) unsigned char sf_raw[];
  T* S = reinterpret_cast<T*>(sf_raw);
  __shared__ int32_t snode[NF];
  __shared__ double ssf[NF];
  const int tid = threadIdx.x;
  const T zero = from_double<T>(0.0);
  for (int i = tid; i < 3 * Sh::kTab; i += NT) S[i] = tabs.tab[i];
  const T *t1 = S, *t2 = S + Sh::kTab, *t3 = S + 2 * Sh::kTab;
  T *M = S + Sh::sM, *X = S + Sh::sX, *A = S + Sh::sA, *C = S + Sh::sC, *U = S + Sh::sU, *R = S + Sh::sR, *U3 = S + Sh::sU3;
  bool bad = false, nonfinite = false;
  for (int item = blockIdx.x; item < cnt; item += gridDim.x) {
    const int e = __ldg(ce + item);
    __syncthreads();  // the previous element's entries have been read (and the tables are in place)
    // coordinates relative to the element's first node: the functions of the value parameters sum to
    // one, so a constant does not change the gradients, and the sums below lose no digits to it
    const int node0 = __ldg(en + (size_t)e * NF);
    const double sf0 = scale ? __ldg(scale + (size_t)e * NF) : 1.0;
    for (int t = tid; t < NF; t += NT) {
      const int pm = __ldg(tabs.param + t), m = pm & 0xffff;
      const int node = __ldg(en + (size_t)e * NF + m);
      const double sf = scale ? __ldg(scale + (size_t)e * NF + m) : 1.0;
      snode[m] = node;
      ssf[m] = sf;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double* xc = coords + (size_t)c * n_nodes;
        const double x = __ldg(xc + node) * sf;
        S[Sh::gx + c * NF + t] = from_double<T>(pm & kSFValue ? x - __ldg(xc + node0) * sf0 : x);
      }
    }
    const double kd = kappa ? __ldg(kappa + e) : 1.0;
    if (!isfinite(kd)) nonfinite = true;
    const T kap = from_double<T>(kd);
    __syncthreads();
    // geometry: xi1 to [c][V, D][f3][f2][q1]
    for (int u = tid; u < 6 * N * N * Q; u += NT) {
      const int q = u % Q, line = (u / Q) % (N * N), cd = u / (Q * N * N), c = cd >> 1;
      const T* tb = t1 + (cd & 1 ? Sh::oD : 0) + q;
      const T* s = S + Sh::gx + c * NF + line * N;
      T v = zero;
#pragma unroll
      for (int f = 0; f < N; ++f) mac(v, s[f], tb[f * Q]);
      finish(v);
      S[Sh::gA + u] = v;
    }
    __syncthreads();
    // xi2 to [c][DV, VD, VV][f3][q2][q1]
    for (int u = tid; u < 9 * N * Q * Q; u += NT) {
      const int q1 = u % Q, q2 = (u / Q) % Q, f3 = (u / (Q * Q)) % N, ck = u / (Q * Q * N), c = ck / 3, k = ck % 3;
      const T* s = S + Sh::gA + ((c * 2 + (k == 0 ? 1 : 0)) * N + f3) * N * Q + q1;
      const T* tb = t2 + (k == 1 ? Sh::oD : 0) + q2;
      T v = zero;
#pragma unroll
      for (int f = 0; f < N; ++f) mac(v, s[f * Q], tb[f * Q]);
      finish(v);
      S[Sh::gB + u] = v;
    }
    __syncthreads();
    // xi3 to J[c * 3 + k][g]
    for (int u = tid; u < 9 * NG; u += NT) {
      const int q12 = u % (Q * Q), q3 = (u / (Q * Q)) % Q, ck = u / NG;
      const T* s = S + Sh::gB + ck * N * Q * Q + q12;
      const T* tb = t3 + (ck % 3 == 2 ? Sh::oD : 0) + q3;
      T v = zero;
#pragma unroll
      for (int f = 0; f < N; ++f) mac(v, s[f * Q * Q], tb[f * Q]);
      finish(v);
      S[Sh::gJ + u] = v;
    }
    __syncthreads();
    for (int g = tid; g < NG; g += NT) {
      T J[3][3];
#pragma unroll
      for (int i = 0; i < 9; ++i) J[i / 3][i % 3] = S[Sh::gJ + i * NG + g];
      const T G00 = J[0][0] * J[0][0] + J[1][0] * J[1][0] + J[2][0] * J[2][0];
      const T G11 = J[0][1] * J[0][1] + J[1][1] * J[1][1] + J[2][1] * J[2][1];
      const T G22 = J[0][2] * J[0][2] + J[1][2] * J[1][2] + J[2][2] * J[2][2];
      const T G01 = J[0][0] * J[0][1] + J[1][0] * J[1][1] + J[2][0] * J[2][1];
      const T G02 = J[0][0] * J[0][2] + J[1][0] * J[1][2] + J[2][0] * J[2][2];
      const T G12 = J[0][1] * J[0][2] + J[1][1] * J[1][2] + J[2][1] * J[2][2];
      const T A00 = G11 * G22 - G12 * G12, A11 = G00 * G22 - G02 * G02, A22 = G00 * G11 - G01 * G01;
      const T A01 = G02 * G12 - G01 * G22, A02 = G01 * G12 - G02 * G11, A12 = G01 * G02 - G00 * G12;
      const T det = G00 * A00 + G01 * A01 + G02 * A02;
      if (!(det > zero)) bad = true;
      // GU * Jacobian * w * kappa = adj(GL) / det * sqrt(det) * w * kappa
      const T sc = kap * wg[g] * tp_rsqrt(det);
      M[g] = A00 * sc; M[NG + g] = A11 * sc; M[2 * NG + g] = A22 * sc;
      M[3 * NG + g] = A01 * sc; M[4 * NG + g] = A02 * sc; M[5 * NG + g] = A12 * sc;
    }
    __syncthreads();
    // stage 1: X0 (M00 DD), X1 (M11 VV), X2 (M22 VV), X12 (M12 VV) [pair][line], X01 (M01 DV), X02 (M02 DV)
    for (int u = tid; u < Sh::kX; u += NT) {
      constexpr int kSym = 4 * NS * Q * Q;
      const int line = u % (Q * Q);
      int mi;
      const T* tb;
      if (u < kSym) {
        const int ty = u / (NS * Q * Q), pr = (u / (Q * Q)) % NS;
        mi = ty == 3 ? 5 : ty;
        tb = t1 + (ty == 0 ? Sh::oDD : Sh::oVV) + pr * Q;
      } else {
        const int v = u - kSym, ty = v / (NA * Q * Q), pr = (v / (Q * Q)) % NA;
        mi = 3 + ty;
        tb = t1 + Sh::oDV + pr * Q;
      }
      T v = zero;
      dot_add<Q>(v, M + mi * NG + line * Q, 1, tb);
      finish(v);
      X[u] = v;
    }
    __syncthreads();
    // stage 2
    constexpr int QQ = Q * Q;
    const T *X0 = X, *X1 = X + NS * QQ, *X2 = X + 2 * NS * QQ, *X12 = X + 3 * NS * QQ, *X01 = X + 4 * NS * QQ,
            *X02 = X01 + NA * QQ;
    for (int u = tid; u < NH * Q; u += NT) {
      const int q3 = u % Q, hp = __ldg(tabs.half + u / Q), i = hp & 0xffff, j = hp >> 16;
      const int a1 = i % N, a2 = i / N, b1 = j % N, b2 = j / N;
      const int s1 = sym_at<N>(a1, b1), s2 = sym_at<N>(a2, b2);
      T v = zero;
      dot_add<Q>(v, X0 + s1 * QQ + q3 * Q, 1, t2 + Sh::oVV + s2 * Q);
      dot_add<Q>(v, X1 + s1 * QQ + q3 * Q, 1, t2 + Sh::oDD + s2 * Q);
      dot_add<Q>(v, X01 + (a1 * N + b1) * QQ + q3 * Q, 1, t2 + Sh::oDV + (b2 * N + a2) * Q);
      dot_add<Q>(v, X01 + (b1 * N + a1) * QQ + q3 * Q, 1, t2 + Sh::oDV + (a2 * N + b2) * Q);
      finish(v);
      A[u] = v;
    }
    for (int u = tid; u < NA * NA * Q; u += NT) {
      const int q3 = u % Q, ij = u / Q, i = ij / NA, j = ij % NA;
      const int a1 = i % N, a2 = i / N, b1 = j % N, b2 = j / N;
      T v = zero;
      dot_add<Q>(v, X02 + (a1 * N + b1) * QQ + q3 * Q, 1, t2 + Sh::oVV + sym_at<N>(a2, b2) * Q);
      dot_add<Q>(v, X12 + sym_at<N>(a1, b1) * QQ + q3 * Q, 1, t2 + Sh::oDV + (a2 * N + b2) * Q);
      finish(v);
      U[u] = v;
    }
    for (int u = tid; u < NS * NS * Q; u += NT) {
      const int q3 = u % Q, s2 = (u / Q) % NS, s1 = u / (Q * NS);
      T v = zero;
      dot_add<Q>(v, X2 + s1 * QQ + q3 * Q, 1, t2 + Sh::oVV + s2 * Q);
      finish(v);
      C[u] = v;
    }
    __syncthreads();
    // stage 3
    for (int u = tid; u < NA * NA * N; u += NT) {  // unit (ij, a3): U3[ij][a3][b3], test value, trial slope
      const int a3 = u % N, ij = u / N;
      T c[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) c[q] = U[ij * Q + q];
#pragma unroll
      for (int b3 = 0; b3 < N; ++b3) {
        T v = zero;
        dot_add<Q>(v, c, 1, t3 + Sh::oDV + (b3 * N + a3) * Q);
        finish(v);
        U3[u * N + b3] = v;
      }
    }
    for (int u = tid; u < NH * 2; u += NT) {  // unit (h, half of the pairs): R[h][s3]
      const int h = u >> 1, hp = __ldg(tabs.half + h), i = hp & 0xffff, j = hp >> 16;
      const int s12 = sym_at<N>(i % N, j % N) * NS + sym_at<N>(i / N, j / N);
      T a[Q], c[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        a[q] = A[h * Q + q];
        c[q] = C[s12 * Q + q];
      }
#pragma unroll
      for (int k = 0; k < NS / 2; ++k) {
        const int s3 = 2 * k + (u & 1);
        T v = zero;
        dot_add<Q>(v, a, 1, t3 + Sh::oVV + s3 * Q);
        dot_add<Q>(v, c, 1, t3 + Sh::oDD + s3 * Q);
        finish(v);
        R[h * NS + s3] = v;
      }
    }
    __syncthreads();
    // entries: K(m, n) = R + U3(m, n) + U3(n, m), scaled by SF(m) SF(n)
    auto entry = [&](const SFPair& pr) {
      T v = R[pr.r] + (U3[pr.ab] + U3[pr.ba]);
      double d = to_double(v);
      if (scale) d = d * ssf[pr.mn & 0xffff] * ssf[pr.mn >> 16];
      return d;
    };
    const int4* plist = reinterpret_cast<const int4*>(tabs.pairs);
    auto pair_at = [&](int t) {
      const int4 q = __ldg(plist + t);
      return SFPair{q.x, q.y, q.z, q.w};
    };
    if (Kel) {
      double* Ke = Kel + (size_t)item * Sh::NP;
      for (int t = tid; t < Sh::NP; t += NT) Ke[t] = entry(pair_at(t));
    } else {
      for (int t0 = tid; t0 < Sh::NP; t0 += kTPScatter * NT)
        scatter_batch(t0, NT, Sh::NP, [&](int t, double& v, long long& pmn, long long& pnm) {
          const SFPair pr = pair_at(t);
          const int m = pr.mn & 0xffff, n = pr.mn >> 16;
          v = entry(pr);
          pmn = entry_pos(slots, e, NF, m, n, rp, ci, snode[m], snode[n] + 1);
          if (m != n) pnm = entry_pos(slots, e, NF, n, m, rp, ci, snode[n], snode[m] + 1);
        }, values, err);
    }
  }
  if (bad) gfe_raise(err, GFE_DEVERR_JACOBIAN);
  if (nonfinite) gfe_raise(err, GFE_DEVERR_NONFINITE);
}

// values += the packed element matrices Kel[item][pair] of one colour's elements (no two share a row).  The colours'
// launches overlap (launch_chained): 36 x 31 x 33 quadratic elements 731 -> 712 us a call.
__global__ void tp_add_element_matrices(const int32_t* __restrict__ ce, int32_t cnt, int32_t nns, int32_t npairs,
                                        const int32_t* __restrict__ en, const SFPair* __restrict__ pairs,
                                        const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                        const int32_t* __restrict__ slots, const double* __restrict__ Kel,
                                        double* __restrict__ values, unsigned* err) {
  const long long total = (long long)cnt * npairs;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x, pmn = -2, pnm = -2;
  double v = 0.0;
  auto load = [&] {
    const int item = (int)(t / npairs), p = (int)(t - (long long)item * npairs);
    const int e = __ldg(ce + item), mn = __ldg(&pairs[p].mn), m = mn & 0xffff, n = mn >> 16;
    v = __ldcs(Kel + t);
    const int rm = __ldg(en + (size_t)e * nns + m), rn = __ldg(en + (size_t)e * nns + n);
    pmn = entry_pos(slots, e, nns, m, n, rp, ci, rm, rn + 1);
    pnm = m == n ? -2 : entry_pos(slots, e, nns, n, m, rp, ci, rn, rm + 1);
  };
  if (t < total) load();
  chain_wait();
  chain_release();
  while (t < total) {
    const double o0 = pmn >= 0 ? __ldcg(values + pmn) : 0.0, o1 = pnm >= 0 ? __ldcg(values + pnm) : 0.0;
    if (pmn >= 0) values[pmn] = o0 + v;
    if (pnm >= 0) values[pnm] = o1 + v;
    if (pmn < 0 || pnm == -1) gfe_raise(err, GFE_DEVERR_SLOT);
    t += (long long)gridDim.x * blockDim.x;
    if (t < total) load();
  }
}

// Number of 1D functions a direction when the sum-factorised kernel takes the basis (3 or 4), else 0: the
// same N in every direction and N Gauss points each (the default rules).  Other rules and mixed orders
// keep the pairwise kernel, and so does FP32, which has not been moved (Q3 24^3 4.34 ms, float-float here 1.57).
int sf_functions(const int32_t* order, const int32_t* ngauss) {
  if (order[0] < 2 || order[0] > 4) return 0;
  const int n = order[0] == 2 ? 3 : 4;
  for (int d = 0; d < 3; ++d)
    if (order[d] < 2 || order[d] > 4 || (order[d] == 2 ? 3 : 4) != n || ngauss[d] != n) return 0;
  return n;
}

template <typename T, int N>
int sf_tables(const int32_t* order, const SFTables<T>** out) {
  using Sh = SFShape<N>;
  constexpr int Q = Sh::Q;
  static std::map<std::array<int, 4>, SFTables<T>> cache;
  int dev = 0;
  GFE_CUDA_TRY(cudaGetDevice(&dev));
  const std::array<int, 4> key = {dev, order[0], order[1], order[2]};
  std::lock_guard<std::mutex> lk(g_tp_mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = &it->second;
    return GFE_OK;
  }
  std::vector<T> tab(3 * Sh::kTab);
  double gx[4], gw[4];
  gauss01(Q, gx, gw);
  for (int d = 0; d < 3; ++d) {
    double V[N][Q], D[N][Q];
    T* o = tab.data() + d * Sh::kTab;
    for (int f = 0; f < N; ++f)
      for (int q = 0; q < Q; ++q) {
        if (order[d] == 4) hermite1d(f / 2, f % 2, gx[q], &V[f][q], &D[f][q]);
        else lagrange1d(order[d], f, gx[q], &V[f][q], &D[f][q]);
        o[f * Q + q] = to_elem<T>(V[f][q]);
        o[Sh::oD + f * Q + q] = to_elem<T>(D[f][q]);
      }
    for (int a = 0; a < N; ++a)
      for (int b = 0; b < N; ++b)
        for (int q = 0; q < Q; ++q) {
          if (a <= b) {
            o[Sh::oVV + sym_pair(a, b, N) * Q + q] = to_elem<T>(V[a][q] * V[b][q]);
            o[Sh::oDD + sym_pair(a, b, N) * Q + q] = to_elem<T>(D[a][q] * D[b][q]);
          }
          o[Sh::oDV + (a * N + b) * Q + q] = to_elem<T>(D[a][q] * V[b][q]);
        }
  }
  // element parameters in Iron's order (local nodes xi1 fastest, then the Hermite directions' derivatives)
  std::vector<int32_t> param(Sh::NF), fn(Sh::NF);
  int nn[3], nder = 1, m = 0;
  for (int d = 0; d < 3; ++d) {
    nn[d] = order[d] == 4 ? 2 : order[d] + 1;
    if (order[d] == 4) nder *= 2;
  }
  for (int a3 = 0; a3 < nn[2]; ++a3)
    for (int a2 = 0; a2 < nn[1]; ++a2)
      for (int a1 = 0; a1 < nn[0]; ++a1)
        for (int k = 0; k < nder; ++k, ++m) {
          const int at[3] = {a1, a2, a3};
          int f[3], bit = 0;
          for (int d = 0; d < 3; ++d) f[d] = order[d] == 4 ? 2 * at[d] + ((k >> bit++) & 1) : at[d];
          fn[m] = f[0] | (f[1] << 4) | (f[2] << 8);
          param[f[0] + N * (f[1] + N * f[2])] = m | (k == 0 ? kSFValue : 0);
        }
  std::vector<int32_t> half;
  for (int i = 0; i < Sh::NA; ++i)
    for (int j = i; j < Sh::NA; ++j) half.push_back(i | (j << 16));
  std::vector<SFPair> pairs;
  for (int a = 0; a < Sh::NF; ++a)
    for (int b = a; b < Sh::NF; ++b) {
      const int i = (fn[a] & 15) + N * ((fn[a] >> 4) & 15), j = (fn[b] & 15) + N * ((fn[b] >> 4) & 15);
      const int a3 = fn[a] >> 8, b3 = fn[b] >> 8;
      const int h = i <= j ? sym_pair(i, j, Sh::NA) : sym_pair(j, i, Sh::NA);
      const int s3 = a3 <= b3 ? sym_pair(a3, b3, N) : sym_pair(b3, a3, N);
      pairs.push_back({a | (b << 16), h * Sh::NS + s3, (i * Sh::NA + j) * Sh::NA + a3 * N + b3,
                       (j * Sh::NA + i) * Sh::NA + b3 * N + a3});
    }
  SFTables<T> t;
  auto up = [](auto** p, const auto& v) -> int {
    GFE_CUDA_TRY(cudaMalloc(p, sizeof(v[0]) * v.size()));
    GFE_CUDA_TRY(cudaMemcpy(*p, v.data(), sizeof(v[0]) * v.size(), cudaMemcpyHostToDevice));
    return GFE_OK;
  };
  int rc;
  if ((rc = up(&t.tab, tab)) || (rc = up(&t.pairs, pairs)) || (rc = up(&t.half, half)) || (rc = up(&t.param, param))) return rc;
  *out = &(cache[key] = t);
  return GFE_OK;
}

// Meshes whose packed element matrices fit kSFScratch form them in one launch over all elements and add
// them colour by colour in small kernels, as a colour alone leaves SMs idle or ends in a nearly empty
// wave; larger ones add straight into the values, one launch a colour.
constexpr size_t kSFScratch = 256u << 20;

template <typename T, int N>
int launch_tp_sf(const int32_t* order, const int32_t* ngauss, int32_t n_nodes, const int32_t* en, const double* coords,
                 const double* scale, const double* kappa, const int32_t* color_elems, const int32_t* color_ptr_host,
                 int32_t n_colors, const int32_t* rp, const int32_t* ci, const int32_t* slots, double* values,
                 cudaStream_t s, int* launches) {
  using Sh = SFShape<N>;
  const TPTables<T>* t = nullptr;  // Gauss weights in the element type
  const SFTables<T>* sf = nullptr;
  if (int rc = tp_tables<T>(order, ngauss, &t)) return rc;
  if (int rc = sf_tables<T, N>(order, &sf)) return rc;
  const int32_t n_elem = n_colors > 0 ? color_ptr_host[n_colors] : 0;
  if (n_elem == 0) return GFE_OK;
  const size_t sm = sizeof(T) * Sh::kShared;
  auto* kernel = laplace_tp_sf_kernel<T, N>;
  GFE_CUDA_TRY(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  unsigned* err = gfe::device_error_word();
  double* Kel = nullptr;
  const size_t bytes = sizeof(double) * (size_t)n_elem * Sh::NP;
  // without the scratch (none is allocated inside a graph capture) the entries are added colour by colour
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  GFE_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
  if (bytes <= kSFScratch && cap == cudaStreamCaptureStatusNone &&
      gfe::scratch_alloc((void**)&Kel, bytes, s, "element matrices"))
    Kel = nullptr;
  auto launch = [&](int c0, int cnt) {
    const int grid = std::min(cnt, 16 * gfe::sm_count());
    kernel<<<grid, Sh::kThreads, sm, s>>>(color_elems + c0, cnt, n_nodes, en, coords, scale, kappa, t->w, *sf, rp, ci,
                                          slots, values, Kel, err);
    ++*launches;
  };
  if (Kel) launch(0, n_elem);
  bool first = true;
  for (int c = 0; c < n_colors; ++c) {
    const int c0 = color_ptr_host[c], cnt = color_ptr_host[c + 1] - c0;
    if (cnt <= 0) continue;
    if (!Kel) {
      launch(c0, cnt);
      continue;
    }
    const int grid = (int)std::min<long long>(((long long)cnt * Sh::NP + 255) / 256, 16ll * gfe::sm_count());
    gfe::launch_chained(!first, tp_add_element_matrices, grid, 256, s, color_elems + c0, cnt, Sh::NF, Sh::NP, en,
                        sf->pairs, rp, ci, slots, Kel + (size_t)c0 * Sh::NP, values, err);
    first = false;
    ++*launches;
  }
  gfe::scratch_free(Kel, s);
  return GFE_OK;
}

}  // namespace
