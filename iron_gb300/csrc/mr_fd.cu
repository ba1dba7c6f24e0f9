// mr_fd.cu -- Iron's finite-difference Jacobian of the Q2/Q1 Mooney-Rivlin element in FP64.
//
// EquationsSet_FiniteElementJacobianEvaluateFD (src/equations_set_routines.F90:2839-2962): the element
// residual R0 at the current parameters, then for every element parameter j (27 nodes of each
// displacement component, then the 8 pressure nodes) the residual with that parameter raised by
// delta = (1 + ||dep||_2) * step, and column j = (R_j - R0) / delta.  ||dep||_2 is the L2 norm of the
// whole dependent parameter vector (DistributedVector_L2Norm).
//
// The kernel is bound by the FP64 pipe.  Raising one displacement parameter changes one row of the
// deformed gradient Z at each Gauss point by a multiple of the node's basis gradient, so a column
// takes the point's stored state (Z, V = Z U^-1, two rows of cofactors, the other entries of Z H Z^T), the
// changed row's products and the stress (about 150 operations a point), the difference of P to its
// unperturbed value, and one sum-factorised transpose (mr_sf.cuh), instead of a whole residual with
// dense tables and the reference metrics again (about 1,650 warp instructions a column; here 220).
// The difference is taken at the Gauss points, before the sum over them.  In a pressure parameter the
// residual is linear, and its difference quotient is formed without the step.
// Measured: 9 x 8 x 7 elements 12.3 -> 0.68 ms (the old kernel ran 63 elements a colour, each warp 23
// residuals in series), error against 64-bit differences 4.5e-13 -> 4.8e-13.
//
// One CTA works on nine columns at a time (three nodes x three components), thread (slot, point):
// 243 of 256 threads.  An element's 27 nodes are split over 1, 3 or 9 CTAs so that small meshes still
// fill the GPU.
#include <algorithm>

#include "gfe_internal.cuh"
#include "mr_sf.cuh"

namespace {

constexpr int NQ = 27, NL = 8, ND = 89;
constexpr int kNormParts = 512;
constexpr int kFDThreads = 256;
constexpr int kSlots = 9;

// partial sums of squares of the dependent vector in a fixed order (kNormParts contiguous chunks)
__global__ void sumsq_parts(const double* __restrict__ v, int64_t n, double* __restrict__ parts) {
  __shared__ double red[256];
  const int64_t chunk = (n + kNormParts - 1) / kNormParts;
  const int64_t a = blockIdx.x * chunk, b = a + chunk < n ? a + chunk : n;
  double s = 0.0;
  for (int64_t i = a + threadIdx.x; i < b; i += blockDim.x) s += v[i] * v[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) parts[blockIdx.x] = red[0];
}

struct FDShared {
  double node[2][81];        // reference and deformed nodes, [c * 27 + n]
  double p[NL];
  double X[243], Z[243];     // gradients [(c * 3 + k) * 27 + g]
  double V[243], cof[243];   // Z U^-1 and cofactors of Z, same layout
  double h[6][NQ], b[6][NQ]; // factor of the reference metric, and Z H Z^T (packed)
  double P0[243];            // unperturbed P / delta, [(k * 3 + c) * 27 + g]
  double iJx[NQ], det[NQ], pg[NQ];
  double A[kSlots][243], B[kSlots][243];  // point differences, transposed stage by stage
  double q[kSlots][NQ], s1[kSlots][18], s2[kSlots][12];
  double tile[ND][kSlots];   // the finished columns of a round
  double v1[3][3], d1[3][3]; // 1D basis values and slopes [node][point]
};

__global__ void __launch_bounds__(kFDThreads, 2)
mr_jacobian_fd_kernel(const int32_t* __restrict__ elems, int32_t count, int32_t parts_per_elem,
                      const int32_t* __restrict__ eq2, const int32_t* __restrict__ elin, int32_t nq2,
                      const double* __restrict__ xg, const double* __restrict__ dep, const double* __restrict__ cpar,
                      const double* __restrict__ norm_parts, double step, const int32_t* __restrict__ slots,
                      double* __restrict__ values, double* __restrict__ Kout, unsigned* err) {
  extern __shared__ double smem[];
  FDShared& S = *reinterpret_cast<FDShared*>(smem);
  const int tid = threadIdx.x, slot = tid / NQ, g = tid % NQ;
  const int item = blockIdx.x / parts_per_elem, part = blockIdx.x % parts_per_elem;
  const int e = __ldg(elems + item);
  const double c1 = cpar[0], c2 = cpar[1];
  auto sync = [] { __syncthreads(); };

  // element data, the step (the parts summed by every thread in one order), 1D tables
  if (tid < NQ) {
    const int n = __ldg(eq2 + (size_t)e * NQ + tid);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      S.node[0][c * NQ + tid] = __ldg(xg + (size_t)c * nq2 + n);
      S.node[1][c * NQ + tid] = dep[(size_t)c * nq2 + n];
    }
  } else if (tid < NQ + NL) {
    S.p[tid - NQ] = dep[(size_t)3 * nq2 + __ldg(elin + (size_t)e * NL + tid - NQ)];
  } else if (tid >= 64 && tid < 73) {
    const int a = (tid - 64) / 3, gp = (tid - 64) % 3;
    const double t = gp == 0 ? -mr_sf::kT : (gp == 1 ? 0.0 : mr_sf::kT), q = gp == 1 ? 0.0 : 0.3;
    S.v1[a][gp] = a == 0 ? q - t : (a == 1 ? 1.0 - 2.0 * q : q + t);
    S.d1[a][gp] = a == 0 ? 4.0 * t - 1.0 : (a == 1 ? -8.0 * t : 4.0 * t + 1.0);
  }
  // ||dep||^2: each warp sums the parts by the same fixed tree
  double ss = 0.0;
  for (int i = tid & 31; i < kNormParts; i += 32) ss += __ldg(norm_parts + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  const double delta = (1.0 + sqrt(ss)) * step, idelta = 1.0 / delta;
  __syncthreads();
  mr_sf::field_gradients(g, slot < 2, S.node[slot & 1], S.A[slot & 1], S.B[slot & 1], slot == 0 ? S.X : S.Z, sync);
  __syncthreads();

  // the unperturbed state of each point
  if (slot == 0) {
    double X[3][3], Z[3][3], h[6], cof[3][3], V[3][3], Y[3][3], b[6];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        X[c][k] = S.X[(c * 3 + k) * NQ + g];
        Z[c][k] = S.Z[(c * 3 + k) * NQ + g];
      }
    const double Jx = mr_sf::geometry(X, h), iJx = 1.0 / Jx;
    const double det = mr_sf::cofactors(Z, cof);
    if (!(det > 0.0 && Jx > 0.0 && isfinite(det))) gfe_raise(err, GFE_DEVERR_JACOBIAN);
    mr_sf::left_metric(Z, h, V, Y, b);
    const double p = mr_sf::point_pressure(g, S.p);
    double sg[6];
    mr_sf::stress(b, fabs(det) * iJx, p, c1, c2, (det > 0.0 ? 1.0 : -1.0) * mr_sf::point_weight(g) * idelta, sg);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double s0 = sg[c == 0 ? 0 : c + 2], s1 = c == 0 ? sg[3] : (c == 1 ? sg[1] : sg[5]);
      const double s2 = c == 0 ? sg[4] : (c == 1 ? sg[5] : sg[2]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        S.P0[(k * 3 + c) * NQ + g] = cof[0][k] * s0 + cof[1][k] * s1 + cof[2][k] * s2;
        S.V[(c * 3 + k) * NQ + g] = V[c][k];
        S.cof[(c * 3 + k) * NQ + g] = cof[c][k];
      }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      S.h[i][g] = h[i];
      S.b[i][g] = b[i];
    }
    S.iJx[g] = iJx;
    S.det[g] = det;
    S.pg[g] = p;
  }
  __syncthreads();

  const int32_t* sl = slots ? slots + (size_t)e * ND * ND : nullptr;
  double* Ke = Kout ? Kout + (size_t)e * ND * ND : nullptr;
  // transposes the nine columns' differences in S.A / S.q and writes them: column of slot s is col(s)
  auto finish_round = [&](int n_slots, auto col) {
    __syncthreads();
    const bool on = slot < n_slots;
    const int s = on ? slot : 0;
    if (on) mr_sf::pressure_t_stage3(g, S.q[s], S.s1[s]);
    int stage = 2;  // of the pressure rows, which share the barriers
    auto next = [&] {
      __syncthreads();
      if (on && stage == 2) mr_sf::pressure_t_stage2(g, S.s1[s], S.s2[s]);
      if (on && stage == 1) mr_sf::pressure_t_stage1(g, S.s2[s], [&](int r, double v) { S.tile[81 + r][s] = v; });
      --stage;
    };
    mr_sf::field_gradients_t(g, on, S.A[s], S.B[s], S.A[s], next, [&](int r, double v) { S.tile[r][s] = v; });
    __syncthreads();
    for (int t = tid; t < ND * n_slots; t += kFDThreads) {
      const int r = t / n_slots, k = t % n_slots, c = col(k);
      const double v = S.tile[r][k];
      if (!isfinite(v)) gfe_raise(err, GFE_DEVERR_NONFINITE);
      if (Ke) Ke[(size_t)r * ND + c] = v;
      if (sl && !(r >= 81 && c >= 81)) {
        const int pos = __ldg(sl + (size_t)r * ND + c);
        if (pos >= 0) values[pos] = __ldcg(values + pos) + v;
        else gfe_raise(err, GFE_DEVERR_SLOT);
      }
    }
  };

  const int per = 9 / parts_per_elem;
  for (int round = part * per; round < (part + 1) * per; ++round) {
    // slot = 3 * (node of the round) + component
    if (slot < kSlots) {
      const int c = slot % 3, ns = round * 3 + slot / 3, ca = c == 2 ? 0 : c + 1, cb = c == 0 ? 2 : c - 1;
      const int a1 = ns % 3, a2 = (ns / 3) % 3, a3 = ns / 9, g1 = g % 3, g2 = (g / 3) % 3, g3 = g / 9;
      const double z0 = S.node[1][c * NQ + ns], d = (z0 + delta) - z0;  // the step as it is taken
      double zc[3], za[3], zb[3], h[6];
      {
        const double v1 = S.v1[a1][g1] * d, v2 = S.v1[a2][g2], v3 = S.v1[a3][g3];
        const double v23 = v2 * v3;
        zc[0] = fma(S.d1[a1][g1] * d, v23, S.Z[(c * 3 + 0) * NQ + g]);
        zc[1] = fma(v1 * v3, S.d1[a2][g2], S.Z[(c * 3 + 1) * NQ + g]);
        zc[2] = fma(v1 * v2, S.d1[a3][g3], S.Z[(c * 3 + 2) * NQ + g]);
      }
#pragma unroll
      for (int i = 0; i < 6; ++i) h[i] = S.h[i][g];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        za[k] = S.Z[(ca * 3 + k) * NQ + g];
        zb[k] = S.Z[(cb * 3 + k) * NQ + g];
      }
      // components in the cyclic order c, ca, cb: cofactor row c is unchanged
      double cof[3][3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int k1 = (k + 1) % 3, k2 = (k + 2) % 3;
        cof[0][k] = S.cof[(c * 3 + k) * NQ + g];
        cof[1][k] = zb[k1] * zc[k2] - zb[k2] * zc[k1];
        cof[2][k] = zc[k1] * za[k2] - zc[k2] * za[k1];
      }
      const double det = mr_sf::dot3(zc, cof[0]);
      if (!(det > 0.0 && isfinite(det))) gfe_raise(err, GFE_DEVERR_JACOBIAN);
      double b[6];
      {
        double vc[3], yc[3], va[3], vb[3];
        mr_sf::row_v(zc, h, vc);
        mr_sf::row_e(vc, h, yc);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          va[k] = S.V[(ca * 3 + k) * NQ + g];
          vb[k] = S.V[(cb * 3 + k) * NQ + g];
        }
        b[0] = mr_sf::dot3(yc, vc);
        b[3] = mr_sf::dot3(yc, va);
        b[4] = mr_sf::dot3(yc, vb);
      }
      b[1] = S.b[ca][g];
      b[2] = S.b[cb][g];
      b[5] = S.b[c == 0 ? 5 : (c == 1 ? 4 : 3)][g];
      const double wd = mr_sf::point_weight(g) * idelta, sgn = det > 0.0 ? 1.0 : -1.0;
      double sg[6];
      mr_sf::stress(b, fabs(det) * S.iJx[g], S.pg[g], c1, c2, sgn * wd, sg);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double* P0 = S.P0 + k * 81 + g;
        double* o = S.A[slot] + k * 81 + g;
        o[c * NQ] = cof[0][k] * sg[0] + cof[1][k] * sg[3] + (cof[2][k] * sg[4] - P0[c * NQ]);
        o[ca * NQ] = cof[0][k] * sg[3] + cof[1][k] * sg[1] + (cof[2][k] * sg[5] - P0[ca * NQ]);
        o[cb * NQ] = cof[0][k] * sg[4] + cof[1][k] * sg[5] + (cof[2][k] * sg[2] - P0[cb * NQ]);
      }
      S.q[slot][g] = wd * (fabs(det) - fabs(S.det[g]));
    }
    finish_round(kSlots, [&](int s) { return (s % 3) * NQ + round * 3 + s / 3; });
  }
  if (part == parts_per_elem - 1) {  // pressure columns: dP/dp_b = w sign(det Z) cof^T psi_b
    if (slot < NL) {
      const double x1 = g % 3 == 0 ? 0.5 - mr_sf::kT : (g % 3 == 1 ? 0.5 : 0.5 + mr_sf::kT);
      const double x2 = (g / 3) % 3 == 0 ? 0.5 - mr_sf::kT : ((g / 3) % 3 == 1 ? 0.5 : 0.5 + mr_sf::kT);
      const double x3 = g / 9 == 0 ? 0.5 - mr_sf::kT : (g / 9 == 1 ? 0.5 : 0.5 + mr_sf::kT);
      const double psi = (slot & 1 ? x1 : 1.0 - x1) * (slot & 2 ? x2 : 1.0 - x2) * (slot & 4 ? x3 : 1.0 - x3);
      const double f = (S.det[g] > 0.0 ? 1.0 : -1.0) * mr_sf::point_weight(g) * psi;
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 3; ++k) S.A[slot][(k * 3 + c) * NQ + g] = f * S.cof[(c * 3 + k) * NQ + g];
      S.q[slot][g] = 0.0;
    }
    finish_round(NL, [&](int s) { return 81 + s; });
  }
}

// values += the element matrices K[e][89][89] of one colour's elements through the slot map (no two
// elements of a colour share a DOF); the pressure-pressure block is not assembled
__global__ void mr_add_element_matrices(const int32_t* __restrict__ elems, int32_t count,
                                        const double* __restrict__ K, const int32_t* __restrict__ slots,
                                        double* __restrict__ values, unsigned* err) {
  constexpr int kEntries = ND * ND;
  const long long n = (long long)count * kEntries;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int pos = -2;  // nothing to add
  double v = 0.0;
  auto load = [&] {
    const int item = (int)(t / kEntries), k = (int)(t % kEntries);
    pos = -2;
    if (k >= 81 * ND && k % ND >= 81) return;
    const size_t at = (size_t)__ldg(elems + item) * kEntries + k;
    pos = __ldg(slots + at);
    v = __ldg(K + at);
  };
  if (t < n) load();
  chain_wait();  // the colours' launches overlap: 9 x 8 x 7 elements 713 -> 680 us a call
  chain_release();
  while (t < n) {
    if (pos >= 0) values[pos] = __ldcg(values + pos) + v;
    else if (pos != -2) gfe_raise(err, GFE_DEVERR_SLOT);
    t += (long long)gridDim.x * blockDim.x;
    if (t < n) load();
  }
}

// Meshes of up to kAllAtOnce elements form all element matrices in one launch, in scratch of at most
// 260 MB (or the caller's K_out), and add them colour by colour in small kernels: a colour of such a
// mesh, an eighth of it, does not fill the GPU (9 x 8 x 7 elements: 63 a colour on 152 SMs).  Larger
// meshes add each round's columns straight into the CSR values, one launch a colour.
constexpr int kAllAtOnce = 4096;

// CTAs an element: enough for four waves of two CTAs an SM, as an element split in n CTAs forms its
// unperturbed state n times (about a tenth of the nine rounds).
int parts_for(int count) {
  const int want = 8 * gfe::sm_count();
  return count >= want ? 1 : (3 * count >= want ? 3 : 9);
}

}  // namespace

extern "C" int gfe_mr_jacobian_fd(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2,
                                  int32_t nlin, const double* xg, const int32_t* color_elems,
                                  const int32_t* color_ptr_host, int32_t n_colors, const double* dep,
                                  const double* cpar, double step, const int32_t* slots, double* values, int64_t nnz,
                                  double* K_out, void* stream) {
  const char* fn = "gfe_mr_jacobian_fd";
  if (n_elem < 0 || nq2 <= 0 || nlin <= 0 || (n_elem > 0 && (!eq2 || !elin || !xg)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid mesh arguments", fn);
  if (!dep || !cpar || !(step > 0.0) || (n_elem > 0 && (!color_elems || !color_ptr_host || n_colors <= 0)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid arguments", fn);
  if (!K_out && (!slots || !values)) return gfe::set_error(GFE_ERR_ARG, "%s: need CSR values + slots or K_out", fn);
  if (color_ptr_host[0] != 0 || color_ptr_host[n_colors] != n_elem)
    return gfe::set_error(GFE_ERR_ARG, "%s: colour offsets must run from 0 to n_elem", fn);
  cudaStream_t s = gfe::as_stream(stream);
  const int64_t ndof = 3ll * nq2 + nlin;
  int rc;
  GFE_CUDA_TRY(cudaFuncSetAttribute((const void*)mr_jacobian_fd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sizeof(FDShared)));
  double* parts = nullptr;
  if ((rc = gfe::scratch_alloc((void**)&parts, sizeof(double) * kNormParts, s, "FD step norm"))) return rc;
  if (values) {
    cudaError_t e = cudaMemsetAsync(values, 0, sizeof(double) * (size_t)nnz, s);
    if (e != cudaSuccess) {
      gfe::scratch_free(parts, s);
      return gfe::set_error(GFE_ERR_CUDA, "%s: %s", fn, cudaGetErrorString(e));
    }
  }
  const bool add = slots && values;
  double* K = K_out;
  bool own = false;
  if (add && !K && n_elem > 0 && n_elem <= kAllAtOnce)
    // without the scratch the columns are added colour by colour, as on larger meshes
    own = gfe::scratch_alloc((void**)&K, sizeof(double) * (size_t)n_elem * ND * ND, s, "FD element matrices") == GFE_OK;
  if (!own) K = K_out;
  unsigned* err = gfe::device_error_word();
  void* prof = gfe::stage_begin(GFE_STAGE_MR_JACOBIAN, s);
  sumsq_parts<<<kNormParts, 256, 0, s>>>(dep, ndof, parts);
  int launches = 1;
  auto launch = [&](int c0, int cnt, const int32_t* sl, double* v) {
    const int pe = parts_for(cnt);
    mr_jacobian_fd_kernel<<<cnt * pe, kFDThreads, sizeof(FDShared), s>>>(color_elems + c0, cnt, pe, eq2, elin, nq2, xg,
                                                                         dep, cpar, parts, step, sl, v, K, err);
    ++launches;
  };
  if (K && n_elem > 0) {
    launch(0, n_elem, nullptr, nullptr);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool chained = cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
    bool first = true;
    for (int c = 0; add && c < n_colors; ++c) {
      const int c0 = color_ptr_host[c], cnt = color_ptr_host[c + 1] - c0;
      if (cnt <= 0) continue;
      const int grid = (int)std::min<long long>(((long long)cnt * ND * ND + 255) / 256, 16ll * gfe::sm_count());
      gfe::launch_chained(!first && chained, mr_add_element_matrices, grid, 256, s, color_elems + c0, cnt, K, slots, values,
                          err);
      first = false;
      ++launches;
    }
  } else {
    for (int c = 0; c < n_colors; ++c) {
      const int c0 = color_ptr_host[c], cnt = color_ptr_host[c + 1] - c0;
      if (cnt > 0) launch(c0, cnt, slots, values);
    }
  }
  gfe::stage_end(GFE_STAGE_MR_JACOBIAN, prof, s, launches);
  if (own) gfe::scratch_free(K, s);
  gfe::scratch_free(parts, s);
  GFE_LAUNCH_CHECK(fn);
  return GFE_OK;
}
