// mr_residual.cu -- Mooney-Rivlin residual and its adjoint for a batch of parameter sets, FP64.
//
// Reference: FiniteElasticity_FiniteElementResidualEvaluate, MOONEY_RIVLIN_SUBTYPE branch
// (src/finite_elasticity_routines.F90:1669-1756), FINITE_ELASTICITY_GAUSS_STRESS_TENSOR (:6985-7061)
// and the element loop of EquationsSet_ResidualEvaluateStaticFEM (src/equations_set_routines.F90:
// 5164-5286).  The adjoint has no counterpart there.
//
// Both kernels are bound by the FP64 pipe.  A CTA takes eight elements, a thread a Gauss point (216
// threads, 96 % of seven warps): gradients and their transposes are sum-factorised (mr_sf.cuh), the
// point formulas work on Z H Z^T and cofactors (no square root, no division but one), and the
// reference metric (a factor of H, J_x) is formed once an element and kept in registers over the parameter sets
// of the CTA's share of the batch.  About 310 FP64 operations a point and parameter set for the
// residual (1,650 warp instructions an element before, with dense tables, pow and divisions) and 520
// for the adjoint.
// Measured, 16^3 elements x 64 sets: residual and adjoint together 56.1 -> 12.8 ms.  Error of an interior
// element's residual against 80-bit arithmetic (1 % perturbed, undeformed mean): 1.0e-13 with the dense
// tables, 2.7e-14 here (node differences are exact, see mr_sf.cuh).
#include <algorithm>

#include "gfe_internal.cuh"
#include "mr_sf.cuh"

namespace {

constexpr int NQ = 27, NL = 8, ND = 89;
constexpr int kElems = 8;
constexpr int kThreads = kElems * NQ;  // 216

// Batches whose element vectors fit kScratchBytes form them in one launch over all elements and add
// them colour by colour in small kernels; a colour alone, an eighth of the mesh, leaves SMs idle or
// ends in a nearly empty wave.  Larger ones add straight into the result, one launch a colour.
constexpr size_t kScratchBytes = 256u << 20;

struct ElemShared {
  double u[81], A[162], B[243], grad[243], p[NL], q[NQ], s1[18], s2[12];
  int dof[ND + 1];
};

// ---- point formulas of the adjoint ----------------------------------------------------------------
// Reverse sweep through P = w sign(det) cof^T sigma, sigma = dev(a1 B^2 + a2 B) + p I, a1 = -2 c2 / J,
// a2 = 2 (c1 + I1 c2) / J, B = J^(-2/3) Z H Z^T, J = |det Z| / J_x, for the cotangent V of P and Vp of
// w (J_z - J_x).  With T = dev of the symmetric part of sigma's cotangent:
//   Bbar = a1 (T B + B T) + a2 T + 2 c2 t2bar I,  t2bar = (T : B) / J,
//   Jbar = -(2/3 Bbar : B + T : S) / J,  detbar = sign (Jbar / J_x + w Vp),
//   Zbar = 2 J^(-2/3) Bbar Z H + detbar cof + the cofactors' cross products.
__device__ __forceinline__ void point_vjp(const double (&Z)[3][3], const double (&h)[6], double iJx, double p, double w,
                                          double c1, double c2, const double (&V)[3][3], double Vp, double (&Zb)[3][3],
                                          double& pb, double& c1b, double& c2b) {
  double cof[3][3], W[3][3], B[6];
  const double det = mr_sf::cofactors(Z, cof);
  const double sgn = det > 0.0 ? 1.0 : -1.0, J = fabs(det) * iJx;
  const double r = rcbrt(J), r2 = r * r, iJ = r2 * r;
  {
    double Vz[3][3], Y[3][3];
    mr_sf::left_metric(Z, h, Vz, Y, B);
#pragma unroll
    for (int i = 0; i < 6; ++i) B[i] *= r2;
#pragma unroll
    for (int c = 0; c < 3; ++c) mr_sf::row_zh(Y[c], h, W[c]);
  }
  const double I1 = B[0] + B[1] + B[2];
  const double a1 = -2.0 * c2 * iJ, a2 = 2.0 * fma(I1, c2, c1) * iJ;
  const double ws = sgn * w;
  // cotangents of sigma (kept as sb + sb^T, packed) and of the cofactors
  double T[6], cb[3][3];
  {
    double sb[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int m = 0; m < 3; ++m)
        sb[c][m] = ws * (cof[c][0] * V[0][m] + cof[c][1] * V[1][m] + cof[c][2] * V[2][m]);
    pb = sb[0][0] + sb[1][1] + sb[2][2];
    const double h = -2.0 / 3.0 * pb;
    T[0] = fma(2.0, sb[0][0], h);
    T[1] = fma(2.0, sb[1][1], h);
    T[2] = fma(2.0, sb[2][2], h);
    T[3] = sb[0][1] + sb[1][0];
    T[4] = sb[0][2] + sb[2][0];
    T[5] = sb[1][2] + sb[2][1];
  }
  {
    double S[6], sg[6];
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
    const double h = fma(-1.0 / 3.0, sg[0] + sg[1] + sg[2], p);
#pragma unroll
    for (int i = 0; i < 6; ++i) sg[i] = ws * (i < 3 ? sg[i] + h : sg[i]);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      cb[0][k] = sg[0] * V[k][0] + sg[3] * V[k][1] + sg[4] * V[k][2];
      cb[1][k] = sg[3] * V[k][0] + sg[1] * V[k][1] + sg[5] * V[k][2];
      cb[2][k] = sg[4] * V[k][0] + sg[5] * V[k][1] + sg[2] * V[k][2];
    }
  }
  // M = (2 T) B; 2 T : B, 2 T : B^2
  double M[3][3];
  const int ix[3][3] = {{0, 3, 4}, {3, 1, 5}, {4, 5, 2}};
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) M[i][j] = T[ix[i][0]] * B[ix[0][j]] + T[ix[i][1]] * B[ix[1][j]] + T[ix[i][2]] * B[ix[2][j]];
  const double tb = 0.5 * (M[0][0] + M[1][1] + M[2][2]);  // T : B
  double tbb = 0.0;                                       // T : B^2
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) tbb = fma(M[i][j], B[ix[i][j]], tbb);
  tbb *= 0.5;
  const double t2b = iJ * tb;
  c1b = 2.0 * t2b;
  c2b = 2.0 * fma(I1, t2b, -iJ * tbb);
  // 2 Bbar, packed
  const double i2 = 4.0 * c2 * t2b;
  double Bb[6];
#pragma unroll
  for (int i = 0; i < 3; ++i) Bb[i] = fma(2.0 * a1, M[i][i], fma(a2, T[i], i2));
  Bb[3] = fma(a1, M[0][1] + M[1][0], a2 * T[3]);
  Bb[4] = fma(a1, M[0][2] + M[2][0], a2 * T[4]);
  Bb[5] = fma(a1, M[1][2] + M[2][1], a2 * T[5]);
  const double bb = Bb[0] * B[0] + Bb[1] * B[1] + Bb[2] * B[2] + 2.0 * (Bb[3] * B[3] + Bb[4] * B[4] + Bb[5] * B[5]);
  const double Jb = -iJ * fma(1.0 / 3.0, bb, fma(a1, tbb, a2 * tb));
  const double db = sgn * fma(Jb, iJx, w * Vp);
#pragma unroll
  for (int i = 0; i < 6; ++i) Bb[i] *= r2;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    Zb[0][k] = fma(db, cof[0][k], Bb[0] * W[0][k] + Bb[3] * W[1][k] + Bb[4] * W[2][k]);
    Zb[1][k] = fma(db, cof[1][k], Bb[3] * W[0][k] + Bb[1] * W[1][k] + Bb[5] * W[2][k]);
    Zb[2][k] = fma(db, cof[2][k], Bb[4] * W[0][k] + Bb[5] * W[1][k] + Bb[2] * W[2][k]);
  }
  // cof[c] = Z[c+1] x Z[c+2]
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int a = (c + 1) % 3, b = (c + 2) % 3;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
      Zb[a][k] += Z[b][k1] * cb[c][k2] - Z[b][k2] * cb[c][k1];
      Zb[b][k] += cb[c][k1] * Z[a][k2] - cb[c][k2] * Z[a][k1];
    }
  }
}

// One CTA: elements [8 group, 8 group + 8) of elems[0..count), parameter sets [b0, b1).  ADJOINT:
// du = v^T dR/d(dep) into R and the element's (c10, c01) cotangents into dc_elem[b][item], else the
// residual into R.  scratch: element vectors [item][b][89] instead of adding into R.
template <bool ADJOINT>
__global__ void __launch_bounds__(kThreads, 2)
mr_residual_kernel(const int32_t* __restrict__ elems, int32_t count, int32_t batch, int32_t chunk,
                   const int32_t* __restrict__ eq2, const int32_t* __restrict__ elin, int32_t nq2, int32_t nlin,
                   const double* __restrict__ xg, const double* __restrict__ dep, const double* __restrict__ cpar,
                   const double* __restrict__ v, double* __restrict__ R, double* __restrict__ scratch,
                   double* __restrict__ dc_elem, int32_t n_elem, int32_t item0, unsigned* err) {
  extern __shared__ double smem[];
  const int le = threadIdx.x / NQ, g = threadIdx.x % NQ;
  ElemShared& S = reinterpret_cast<ElemShared*>(smem)[le];
  double* cb_all = smem + sizeof(ElemShared) / sizeof(double) * kElems;  // [8][2][27]
  const int n_chunks = (batch + chunk - 1) / chunk;
  const int group = blockIdx.x / n_chunks, b0 = (blockIdx.x % n_chunks) * chunk, b1 = min(batch, b0 + chunk);
  const int item = group * kElems + le;
  const bool on = item < count;
  const int64_t ndof = 3ll * nq2 + nlin;
  auto sync = [] { __syncthreads(); };
  int node = 0, pnode = 0;
  double zn[3] = {0.0, 0.0, 0.0}, pn = 0.0;
  // node values of parameter set b of the field f ([batch][ndof]), ahead of their use
  auto fetch = [&](const double* f, int b) {
    if (on) {
      const double* d = f + b * ndof;
#pragma unroll
      for (int c = 0; c < 3; ++c) zn[c] = __ldg(d + (size_t)c * nq2 + node);
      if (g < NL) pn = __ldg(d + (size_t)3 * nq2 + pnode);
    }
  };
  auto stage = [&] {
    if (on) {
#pragma unroll
      for (int c = 0; c < 3; ++c) S.u[c * NQ + g] = zn[c];
      if (g < NL) S.p[g] = pn;
    }
  };
  if (on) {
    const int e = __ldg(elems + item);
    node = __ldg(eq2 + (size_t)e * NQ + g);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      S.u[c * NQ + g] = __ldg(xg + (size_t)c * nq2 + node);
      S.dof[c * NQ + g] = c * nq2 + node;
    }
    if (g < NL) {
      pnode = __ldg(elin + (size_t)e * NL + g);
      S.dof[81 + g] = 3 * nq2 + pnode;
    }
  }
  fetch(dep, b0);
  sync();
  double h[6], Jx, iJx;
  {
    double X[3][3];
    mr_sf::field_gradients(g, on, S.u, S.A, S.B, S.grad, sync);
    sync();
#pragma unroll
    for (int i = 0; i < 9; ++i) X[i / 3][i % 3] = S.grad[i * NQ + g];
    Jx = mr_sf::geometry(X, h);
    iJx = 1.0 / Jx;
  }
  const double w = mr_sf::point_weight(g);
  bool bad = false, nonfinite = false;
  for (int b = b0; b < b1; ++b) {
    stage();
    if (ADJOINT) fetch(v, b);
    else if (b + 1 < b1) fetch(dep, b + 1);
    sync();
    mr_sf::field_gradients(g, on, S.u, S.A, S.B, S.grad, sync);
    sync();
    double Z[3][3];
#pragma unroll
    for (int i = 0; i < 9; ++i) Z[i / 3][i % 3] = S.grad[i * NQ + g];
    const double p = mr_sf::point_pressure(g, S.p);
    const double c1 = __ldg(cpar + 2 * b), c2 = __ldg(cpar + 2 * b + 1);
    if constexpr (!ADJOINT) {
      double cof[3][3], V[3][3], Y[3][3], bq[6], sg[6];
      const double det = mr_sf::cofactors(Z, cof);
      if (on && !(det > 0.0 && Jx > 0.0 && isfinite(det))) bad = true;
      mr_sf::left_metric(Z, h, V, Y, bq);
      mr_sf::stress(bq, fabs(det) * iJx, p, c1, c2, det > 0.0 ? w : -w, sg);
      sync();  // grad has been read
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        S.grad[(k * 3 + 0) * NQ + g] = cof[0][k] * sg[0] + cof[1][k] * sg[3] + cof[2][k] * sg[4];
        S.grad[(k * 3 + 1) * NQ + g] = cof[0][k] * sg[3] + cof[1][k] * sg[1] + cof[2][k] * sg[5];
        S.grad[(k * 3 + 2) * NQ + g] = cof[0][k] * sg[4] + cof[1][k] * sg[5] + cof[2][k] * sg[2];
      }
      S.q[g] = w * (fabs(det) - Jx);
    } else {
      sync();  // u, p and grad have been read
      stage();
      if (b + 1 < b1) fetch(dep, b + 1);
      sync();
      mr_sf::field_gradients(g, on, S.u, S.A, S.B, S.grad, sync);
      sync();
      double V[3][3], Zb[3][3], pb, c1b, c2b;
#pragma unroll
      for (int i = 0; i < 9; ++i) V[i % 3][i / 3] = S.grad[i * NQ + g];
      const double Vp = mr_sf::point_pressure(g, S.p);
      point_vjp(Z, h, iJx, p, w, c1, c2, V, Vp, Zb, pb, c1b, c2b);
      sync();
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) S.grad[(k * 3 + c) * NQ + g] = Zb[c][k];
      S.q[g] = pb;
      cb_all[le * 54 + g] = c1b;
      cb_all[le * 54 + 27 + g] = c2b;
    }
    sync();
    double* Rb = R + b * ndof;
    double* Sb = scratch ? scratch + ((size_t)(item0 + item) * batch + b) * ND : nullptr;
    auto out = [&](int i, double val) {
      if (!isfinite(val)) nonfinite = true;
      if (Sb) Sb[i] = val;
      else Rb[S.dof[i]] += val;
    };
    if (on) mr_sf::pressure_t_stage3(g, S.q, S.s1);
    int st = 2;
    auto next = [&] {
      __syncthreads();
      if (on && st == 2) mr_sf::pressure_t_stage2(g, S.s1, S.s2);
      if (on && st == 1) mr_sf::pressure_t_stage1(g, S.s2, [&](int i, double val) { out(81 + i, val); });
      --st;
    };
    mr_sf::field_gradients_t(g, on, S.grad, S.B, S.A, next, out);
    if (ADJOINT && threadIdx.x < 2 * kElems) {
      const int l = threadIdx.x >> 1, it = group * kElems + l;
      const double* s = cb_all + l * 54 + (threadIdx.x & 1) * 27;
      double t = 0.0;
#pragma unroll 9
      for (int i = 0; i < NQ; ++i) t += s[i];
      if (it < count) dc_elem[((size_t)b * n_elem + item0 + it) * 2 + (threadIdx.x & 1)] = t;
    }
    // the next set's stage() writes u and p, last read before the barriers above
  }
  if (bad) gfe_raise(err, GFE_DEVERR_JACOBIAN);
  if (nonfinite) gfe_raise(err, GFE_DEVERR_NONFINITE);
}

// R[b][dof] += element vectors of one colour's items (no two of its elements share a DOF)
__global__ void mr_add_element_vectors(const int32_t* __restrict__ elems, int32_t item0, int32_t count, int32_t batch,
                                       const int32_t* __restrict__ eq2, const int32_t* __restrict__ elin, int32_t nq2,
                                       int64_t ndof, const double* __restrict__ vec, double* __restrict__ R) {
  const long long n = (long long)count * batch * ND;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t at = 0;
  double v = 0.0;
  auto load = [&] {
    const int r = (int)(t % ND);
    const long long ib = t / ND;
    const int item = (int)(ib / batch), b = (int)(ib % batch);
    const int e = __ldg(elems + item);
    const int64_t dof = r < 81 ? (int64_t)(r / NQ) * nq2 + __ldg(eq2 + (size_t)e * NQ + r % NQ)
                               : 3ll * nq2 + __ldg(elin + (size_t)e * NL + r - 81);
    at = b * ndof + dof;
    v = __ldcs(vec + ((size_t)item0 * batch) * ND + t);
  };
  if (t < n) load();
  chain_wait();  // the colours' launches overlap
  chain_release();
  while (t < n) {
    R[at] = __ldcg(R + at) + v;
    t += (long long)gridDim.x * blockDim.x;
    if (t < n) load();
  }
}

// dc[b][q] = sum over the elements in a fixed tree order: one CTA a parameter set
__global__ void __launch_bounds__(256)
sum_dc(const double* __restrict__ dc_elem, int32_t n_elem, double* __restrict__ dc) {
  __shared__ double red[256];
  const int b = blockIdx.x, q = threadIdx.x & 1;
  double s = 0.0;
  for (int e = threadIdx.x >> 1; e < n_elem; e += 128) s += dc_elem[((size_t)b * n_elem + e) * 2 + q];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o >= 2; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x < 2) dc[b * 2 + threadIdx.x] = red[threadIdx.x];
}

size_t shared_bytes(bool adjoint) {
  return sizeof(ElemShared) * kElems + (adjoint ? sizeof(double) * 54 * kElems : 0);
}

// Launches over the batch: all elements at once into scratch, then the colours' additions, or colour by colour.
template <bool ADJOINT>
int run_batch(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin, const double* xg,
              const int32_t* color_elems, const int32_t* color_ptr_host, int32_t n_colors, int32_t batch,
              const double* dep, const double* cpar, const double* v, double* R, double* dc_elem, cudaStream_t s,
              int* launches) {
  const int64_t ndof = 3ll * nq2 + nlin;
  const size_t sm = shared_bytes(ADJOINT);
  GFE_CUDA_TRY(cudaFuncSetAttribute((const void*)mr_residual_kernel<ADJOINT>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  unsigned* err = gfe::device_error_word();
  const size_t bytes = sizeof(double) * (size_t)n_elem * batch * ND;
  double* vec = nullptr;
  // without the scratch (none is allocated inside a graph capture) the entries are added colour by colour
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  GFE_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
  if (n_elem > 0 && bytes <= kScratchBytes && cap == cudaStreamCaptureStatusNone &&
      gfe::scratch_alloc((void**)&vec, bytes, s, "element residuals"))
    vec = nullptr;
  auto launch = [&](int c0, int cnt) {
    const int groups = (cnt + kElems - 1) / kElems;
    // parameter sets a CTA: the metrics are formed once for them (a third of a pass), but at least
    // eight waves of CTAs
    const int chunk = (int)std::max<long long>(1, std::min<long long>(8, (long long)groups * batch / (24ll * gfe::sm_count())));
    const long long grid = (long long)groups * ((batch + chunk - 1) / chunk);
    mr_residual_kernel<ADJOINT><<<(unsigned)grid, kThreads, sm, s>>>(color_elems + c0, cnt, batch, chunk, eq2, elin,
                                                                     nq2, nlin, xg, dep, cpar, v, R, vec, dc_elem,
                                                                     n_elem, c0, err);
    ++*launches;
  };
  if (vec) launch(0, n_elem);
  bool first = true;
  for (int c = 0; c < n_colors; ++c) {
    const int c0 = color_ptr_host[c], cnt = color_ptr_host[c + 1] - c0;
    if (cnt <= 0) continue;
    if (!vec) {
      launch(c0, cnt);
      continue;
    }
    const int grid = (int)std::min<long long>(((long long)cnt * batch * ND + 255) / 256, 16ll * gfe::sm_count());
    gfe::launch_chained(!first, mr_add_element_vectors, grid, 256, s, color_elems + c0, c0, cnt, batch, eq2, elin, nq2, ndof,
                        vec, R);
    first = false;
    ++*launches;
  }
  gfe::scratch_free(vec, s);
  return GFE_OK;
}

int check_mesh(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin, const double* xg,
               const char* fn) {
  if (n_elem < 0 || nq2 <= 0 || nlin <= 0 || (n_elem > 0 && (!eq2 || !elin || !xg)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid mesh arguments", fn);
  return GFE_OK;
}

}  // namespace

extern "C" int gfe_mr_residual(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin,
                               const double* xg, const int32_t* color_elems, const int32_t* color_ptr_host,
                               int32_t n_colors, int32_t batch, const double* dep, const double* cpar, double* R,
                               void* stream) {
  const char* fn = "gfe_mr_residual";
  int rc = check_mesh(n_elem, eq2, elin, nq2, nlin, xg, fn);
  if (rc) return rc;
  if (batch <= 0 || !dep || !cpar || !R || (n_elem > 0 && (!color_elems || !color_ptr_host || n_colors <= 0)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid arguments", fn);
  if (color_ptr_host[0] != 0 || color_ptr_host[n_colors] != n_elem)
    return gfe::set_error(GFE_ERR_ARG, "%s: colour offsets must run from 0 to n_elem", fn);
  cudaStream_t s = gfe::as_stream(stream);
  const int64_t ndof = 3ll * nq2 + nlin;
  GFE_CUDA_TRY(cudaMemsetAsync(R, 0, sizeof(double) * ndof * batch, s));
  void* prof = gfe::stage_begin(GFE_STAGE_MR_RESIDUAL, s);
  int launches = 0;
  rc = run_batch<false>(n_elem, eq2, elin, nq2, nlin, xg, color_elems, color_ptr_host, n_colors, batch, dep, cpar,
                        nullptr, R, nullptr, s, &launches);
  gfe::stage_end(GFE_STAGE_MR_RESIDUAL, prof, s, launches);
  if (rc) return rc;
  GFE_LAUNCH_CHECK(fn);
  return GFE_OK;
}

extern "C" int gfe_mr_residual_vjp(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2,
                                   int32_t nlin, const double* xg, const int32_t* color_elems,
                                   const int32_t* color_ptr_host, int32_t n_colors, int32_t batch, const double* dep,
                                   const double* cpar, const double* v, double* du, double* dc, void* stream) {
  const char* fn = "gfe_mr_residual_vjp";
  int rc = check_mesh(n_elem, eq2, elin, nq2, nlin, xg, fn);
  if (rc) return rc;
  if (batch <= 0 || !dep || !cpar || !v || !du || !dc || (n_elem > 0 && (!color_elems || !color_ptr_host)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid arguments", fn);
  if (color_ptr_host[0] != 0 || color_ptr_host[n_colors] != n_elem)
    return gfe::set_error(GFE_ERR_ARG, "%s: colour offsets must run from 0 to n_elem", fn);
  cudaStream_t s = gfe::as_stream(stream);
  const int64_t ndof = 3ll * nq2 + nlin;
  GFE_CUDA_TRY(cudaMemsetAsync(du, 0, sizeof(double) * ndof * batch, s));
  double* dc_elem = nullptr;
  if ((rc = gfe::scratch_alloc((void**)&dc_elem, sizeof(double) * 2 * (size_t)n_elem * batch, s, "vjp partials")))
    return rc;
  int launches = 0;
  rc = run_batch<true>(n_elem, eq2, elin, nq2, nlin, xg, color_elems, color_ptr_host, n_colors, batch, dep, cpar, v, du,
                       dc_elem, s, &launches);
  if (!rc) sum_dc<<<batch, 256, 0, s>>>(dc_elem, n_elem, dc);
  gfe::scratch_free(dc_elem, s);
  if (rc) return rc;
  GFE_LAUNCH_CHECK(fn);
  return GFE_OK;
}
