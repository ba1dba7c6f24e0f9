// mr.cu -- K5: Mooney-Rivlin (mixed u-p, triquadratic u + trilinear p) Jacobians: FP32 Gauss-point and
// contraction kernels (CUDA cores and tcgen05), the slot map, the row-owning assembly and the entry
// points.  FP64 element matrices are formed by mr_jac64.cu, the residual and its adjoint by
// mr_residual.cu, Iron's finite-difference Jacobian by mr_fd.cu.
//
// Reference: FiniteElasticity_GaussDeformationGradientTensor
// (src/finite_elasticity_routines.F90:5148-5215) with the material frame of
// Coordinates_MaterialSystemCalculate (src/coordinate_routines.F90:3841-3947),
// FiniteElasticity_FiniteElementJacobianEvaluate (:1016-1274) and
// FINITE_ELASTICITY_GAUSS_ELASTICITY_TENSOR (:649-795).
//
// Field layout (Iron's separated component order): the dependent vector holds the deformed
// positions z1, z2, z3 over the n_q2 quadratic nodes followed by the pressure over the n_lin
// linear (corner) nodes; the geometric field x is [3][n_q2].  Element DOF order: 27 z1, 27 z2,
// 27 z3, 8 p (Iron's element parameter order, local nodes xi1 fastest).
#include <climits>
#include <mutex>
#include <type_traits>

#include "df.cuh"
#include "gfe_internal.cuh"
#include "mr_jac64.cuh"
#include "mr_point.cuh"
#include "tcgen05.cuh"

namespace {

// 16-byte multiple in size, so that a TMA bulk copy can stage the whole table
template <typename S>
struct alignas(16) TablesT {
  S dphi[NG][3][NQ];  // d phi_ns / d xi_k at Gauss point g (quadratic basis)
  S w[NG];
  S psi[NG][NL];      // linear basis values at the Gauss points
};
using Tables = TablesT<double>;
using TablesF = TablesT<float>;  // FP32 copy read by the FP32 Gauss-point kernel

// Host construction of the tables (Gauss-Legendre 3-point rule on [0,1], Lagrange bases),
// src/basis_routines.F90:3720-4090, 6804-6890, 7969-8090.
void build_tables(Tables& t) {
  const double s = std::sqrt(0.6);
  const double gx[3] = {(-s + 1.0) / 2.0, 0.5, (s + 1.0) / 2.0};
  const double gw[3] = {2.5 / 9.0, 4.0 / 9.0, 2.5 / 9.0};
  auto q = [](int a, int d, double x) {
    if (d == 0) return a == 0 ? 1.0 - 3.0 * x + 2.0 * x * x : (a == 1 ? 4.0 * x * (1.0 - x) : x * (x + x - 1.0));
    return a == 0 ? 4.0 * x - 3.0 : (a == 1 ? 4.0 - 8.0 * x : 4.0 * x - 1.0);
  };
  auto l = [](int a, double x) { return a == 0 ? 1.0 - x : x; };
  for (int g3 = 0; g3 < 3; ++g3)
    for (int g2 = 0; g2 < 3; ++g2)
      for (int g1 = 0; g1 < 3; ++g1) {
        const int g = g1 + 3 * (g2 + 3 * g3);
        const double xg[3] = {gx[g1], gx[g2], gx[g3]};
        t.w[g] = gw[g1] * gw[g2] * gw[g3];
        for (int a3 = 0; a3 < 3; ++a3)
          for (int a2 = 0; a2 < 3; ++a2)
            for (int a1 = 0; a1 < 3; ++a1) {
              const int ns = a1 + 3 * (a2 + 3 * a3);
              const int ai[3] = {a1, a2, a3};
              for (int k = 0; k < 3; ++k) {
                double v = 1.0;
                for (int d = 0; d < 3; ++d) v *= q(ai[d], d == k ? 1 : 0, xg[d]);
                t.dphi[g][k][ns] = v;
              }
            }
        for (int b3 = 0; b3 < 2; ++b3)
          for (int b2 = 0; b2 < 2; ++b2)
            for (int b1 = 0; b1 < 2; ++b1) t.psi[g][b1 + 2 * (b2 + 2 * b3)] = l(b1, xg[0]) * l(b2, xg[1]) * l(b3, xg[2]);
      }
}

std::mutex g_tab_mu;
Tables* g_tables[64] = {nullptr};

int device_tables(const Tables** out) {
  int dev = 0;
  GFE_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_tab_mu);
  if (!g_tables[dev]) {
    Tables h;
    build_tables(h);
    void* p = nullptr;
    GFE_CUDA_TRY(cudaMalloc(&p, sizeof(Tables)));
    GFE_CUDA_TRY(cudaMemcpy(p, &h, sizeof(Tables), cudaMemcpyHostToDevice));
    g_tables[dev] = static_cast<Tables*>(p);
  }
  *out = g_tables[dev];
  return GFE_OK;
}

TablesF* g_tables_f[64] = {nullptr};

int device_tables_f(const TablesF** out) {
  int dev = 0;
  GFE_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_tab_mu);
  if (!g_tables_f[dev]) {
    Tables h;
    build_tables(h);
    TablesF f;
    for (int g = 0; g < NG; ++g) {
      f.w[g] = (float)h.w[g];
      for (int k = 0; k < 3; ++k)
        for (int n = 0; n < NQ; ++n) f.dphi[g][k][n] = (float)h.dphi[g][k][n];
      for (int m = 0; m < NL; ++m) f.psi[g][m] = (float)h.psi[g][m];
    }
    void* p = nullptr;
    GFE_CUDA_TRY(cudaMalloc(&p, sizeof(TablesF)));
    GFE_CUDA_TRY(cudaMemcpy(p, &f, sizeof(TablesF), cudaMemcpyHostToDevice));
    g_tables_f[dev] = static_cast<TablesF*>(p);
  }
  *out = g_tables_f[dev];
  return GFE_OK;
}

template <typename S>
__device__ __forceinline__ bool gauss_point(const TablesT<S>& T, int g, const S* sz, const S* sx, const S* sp,
                                            GPT<S>& o) {
  S Z[3][3], X[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      S a = S(0), b = S(0);
#pragma unroll 9
      for (int ns = 0; ns < NQ; ++ns) {
        const S d = T.dphi[g][k][ns];
        a += d * sz[c * NQ + ns];
        b += d * sx[c * NQ + ns];
      }
      Z[c][k] = a;
      X[c][k] = b;
    }
  const S dz = point_frame(Z, X, o);
  S p = S(0);
#pragma unroll
  for (int m = 0; m < NL; ++m) p += T.psi[g][m] * sp[m];
  o.p = p;
  o.w = T.w[g];
  return dz > S(0) && o.Jx > S(0) && isfinite(dz);
}

// slot map: for each element and each (r, c), the 0-based CSR position of (dof_r, dof_c); -1 when
// absent, at slots[(e * 89 + r) * 89 + c] (element number e).  One warp per (element, row).
__global__ void mr_slot_kernel(const int32_t* __restrict__ elems, int32_t count, const int32_t* __restrict__ eq2,
                               const int32_t* __restrict__ elin, int32_t nq2, const int32_t* __restrict__ rp,
                               const int32_t* __restrict__ ci, int32_t* __restrict__ slots) {
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; wid < (long long)count * ND;
       wid += nw) {
    const int item = (int)(wid / ND), r = (int)(wid % ND);
    const int e = elems[item];
    auto dof = [&](int i) {
      return i < 81 ? (i / NQ) * nq2 + eq2[(size_t)e * NQ + i % NQ] : 3 * nq2 + elin[(size_t)e * NL + i - 81];
    };
    const int row = dof(r);
    const int lo0 = rp[row] - 1, hi0 = rp[row + 1] - 1;
    for (int c = lane; c < ND; c += 32) {
      const int col = dof(c) + 1;
      int lo = lo0, hi = hi0;
      while (lo < hi) {
        const int mid = lo + ((hi - lo) >> 1);  // no int32 overflow past 2^30 entries
        if (ci[mid] < col) lo = mid + 1; else hi = mid;
      }
      slots[((size_t)e * ND + r) * ND + c] = (lo < hi0 && ci[lo] == col) ? lo : -1;
    }
  }
}

// ----------------------------------------------------------------------------------------------
// Row-owning assembly of element matrices (replaces EquationsMatrices_JacobianElementAdd,
// src/equations_matrices_routines.F90:2866-2909, for a whole mesh at once)
// ----------------------------------------------------------------------------------------------
// The element matrices of all elements are first written to Kel[e][89][89]; then each CSR row is
// summed once from the element rows of the elements around its node, in ascending element order,
// in shared memory, and written out exactly once with coalesced stores.  Each element row and its
// slot-map row are read once, contiguously.  Node incidence: for node k (quadratic nodes 0..nq2-1,
// then linear nodes nq2 + l) up to kMaxInc entries (e * 64 + local index; local 0..26 quadratic,
// 27..34 linear), sorted by element.
// FP32 element matrices lie kKelF floats apart (a 16-byte multiple: they leave by TMA), FP64 ones 89 * 89.
constexpr int kKelF = (ND * ND + 3) / 4 * 4;
template <typename TS>
constexpr int kKelStride = std::is_same<TS, float>::value ? kKelF : ND * ND;
constexpr int kMaxInc = 16;       // elements around one node (8 on a hexahedral grid)
constexpr int kRowWarps = 8;      // warps (rows in flight) per CTA of mr_row_gather_kernel
constexpr int kMaxRowLen = 512;   // entries of one Jacobian row (at most 402 on a regular Q2/Q1 grid)

__global__ void mr_incidence_fill(const int32_t* __restrict__ elems, int32_t count, const int32_t* __restrict__ eq2,
                                  const int32_t* __restrict__ elin, int32_t nq2, int32_t* __restrict__ cnt,
                                  int32_t* __restrict__ list, unsigned* err) {
  const long long n = (long long)count * (NQ + NL);
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int item = (int)(t / (NQ + NL)), loc = (int)(t % (NQ + NL));
    const int e = __ldg(elems + item);
    const int node = loc < NQ ? __ldg(eq2 + (size_t)e * NQ + loc) : nq2 + __ldg(elin + (size_t)e * NL + loc - NQ);
    const int k = atomicAdd(cnt + node, 1);
    if (k < kMaxInc) list[(size_t)node * kMaxInc + k] = e * 64 + loc;
    else gfe_raise(err, GFE_DEVERR_SLOT);
  }
}

// sort each node's incidence list by element (insertion sort of at most kMaxInc entries)
__global__ void mr_incidence_sort(int32_t n_nodes, const int32_t* __restrict__ cnt, int32_t* __restrict__ list) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n_nodes; k += gridDim.x * blockDim.x) {
    int32_t* L = list + (size_t)k * kMaxInc;
    const int m = min(cnt[k], kMaxInc);
    for (int i = 1; i < m; ++i) {
      const int32_t v = L[i];
      int j = i - 1;
      while (j >= 0 && L[j] > v) {
        L[j + 1] = L[j];
        --j;
      }
      L[j + 1] = v;
    }
  }
}

// One warp per CSR row: values[row] = sum over the elements around the row's node of their element
// rows, through the slot map (element number order).  Rows of displacement component mh take local
// row mh * 27 + node index; pressure rows local row 81 + corner index.  The pressure-pressure block
// is not assembled (zero in Iron's matrix).  Every entry of every row is written, so the values
// need no zeroing first.  FP32 element matrices are summed in FP32 (at most 8 terms an entry,
// against the 5e-6 of their own contraction) and widened exactly with integer operations: the FP64 additions and
// conversions kept the FP64 pipe 77 % busy and bounded the kernel.
//
// DRAM bounds it (element matrices and slot map read once, values written once); the instructions come second, so a
// row takes its elements four, two or one at a time (a node has 1, 2, 4 or 8), 32-bit offsets and 16-byte stores, which
// the row's place in shared memory is shifted for: 794 -> 705 us at 32^3 (3.4 GB).  Additions without a branch to a
// spare entry, or that skip absent elements of a fixed group of four, were slower (820, 768 us).
__device__ __forceinline__ double widen(float f) {  // as f32_to_f64_exact, with one rare branch: 734 -> 705 us
  const unsigned u = __float_as_uint(f), t = u & 0x7fffffffu;
  if (t - 0x00800000u >= 0x7f000000u && t != 0u) return (double)f;  // subnormal, infinite or NaN
  const unsigned hi = t == 0u ? 0u : (t >> 3) + (896u << 20);
  return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)(u << 29));
}
__device__ __forceinline__ double widen(double f) { return f; }

template <int G, typename TS>
__device__ __forceinline__ bool add_element_rows(TS* B, int r0, int len, int list, int i, int mh,
                                                 const TS* __restrict__ Kel, const int32_t* __restrict__ slots) {
  const int lane = threadIdx.x & 31;
  int at[G][3];  // place in the row; INT_MIN: nothing to add, else outside it: a wrong slot
  TS val[G][3];
  bool ok = true;
  // every load of the group is issued before its additions, which then run in ascending element order
#pragma unroll
  for (int u = 0; u < G; ++u) {
    const int packed = __shfl_sync(0xffffffffu, list, i + u);
    const int e = packed >> 6, loc = packed & 63;
    const int lr = loc < NQ ? mh * NQ + loc : 81 + loc - NQ;
    const int32_t* srow = slots + ((size_t)e * (ND * ND) + lr * ND) + lane;
    const TS* krow = Kel + ((size_t)e * kKelStride<TS> + lr * ND) + lane;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const bool in = j < 2 || lane + 64 < (lr >= 81 ? 81 : ND);
      at[u][j] = in ? __ldg(srow + 32 * j) - r0 : INT_MIN;
      val[u][j] = in ? __ldg(krow + 32 * j) : TS(0);
    }
  }
#pragma unroll
  for (int u = 0; u < G; ++u) {
    // an element row's columns are distinct: its loads need not wait for its stores
    bool inside[3];
    TS sum[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      inside[j] = (unsigned)at[u][j] < (unsigned)len;
      ok &= inside[j] || at[u][j] == INT_MIN;
      sum[j] = (inside[j] ? B[at[u][j]] : TS(0)) + val[u][j];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (inside[j]) B[at[u][j]] = sum[j];
    __syncwarp();  // the next element may add to the same entries
  }
  return ok;
}

template <typename TS>
__global__ void __launch_bounds__(kRowWarps * 32, sizeof(TS) == 4 ? 5 : 4)
mr_row_gather_kernel(int32_t nq2, int32_t nlin, const int32_t* __restrict__ cnt, const int32_t* __restrict__ list,
                     const TS* __restrict__ Kel, const int32_t* __restrict__ slots, const int32_t* __restrict__ rp,
                     double* __restrict__ values, unsigned* err) {
  __shared__ __align__(16) TS buf[kRowWarps][kMaxRowLen + 4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n_rows = 3 * nq2 + nlin, step = gridDim.x * kRowWarps;
  // what a row needs to start (its bounds and its node's elements, a lane an entry), loaded one row ahead
  struct Head {
    int mh, r0, r1, m, list;
  };
  static_assert(kMaxInc <= 32, "a lane an element");
  auto head = [&](int row) {
    Head h;
    h.mh = row < 3 * nq2 ? (row >= nq2) + (row >= 2 * nq2) : 0;
    const int node = row < 3 * nq2 ? row - h.mh * nq2 : nq2 + row - 3 * nq2;
    h.r0 = __ldg(rp + row) - 1;
    h.r1 = __ldg(rp + row + 1) - 1;
    h.m = min(__ldg(cnt + node), kMaxInc);
    h.list = lane < kMaxInc ? __ldg(list + (size_t)node * kMaxInc + lane) : 0;
    return h;
  };
  Head next{};
  if (blockIdx.x * kRowWarps + w < n_rows) next = head(blockIdx.x * kRowWarps + w);
  for (int row = blockIdx.x * kRowWarps + w; row < n_rows; row += step) {
    const Head h = next;
    if (row + step < n_rows) next = head(row + step);
    const int r0 = h.r0, len = h.r1 - r0, m = h.m, mh = h.mh;
    bool ok = len <= kMaxRowLen;
    if (!ok) {
      gfe_raise(err, GFE_DEVERR_SLOT);
      continue;
    }
    // entry o of the row is B[o]; B - shift is 16-byte aligned and so is its place in `values`
    double* out = values + r0;
    const int shift = (int)((reinterpret_cast<uintptr_t>(out) >> 3) & 1);
    TS* B = buf[w] + shift;
    for (int j = lane * 2; j < len + shift; j += 64) buf[w][j] = buf[w][j + 1] = TS(0);
    __syncwarp();
    int i = 0;
    for (; m - i >= 4; i += 4) ok &= add_element_rows<4>(B, r0, len, h.list, i, mh, Kel, slots);
    if (m & 2) ok &= add_element_rows<2>(B, r0, len, h.list, i, mh, Kel, slots);
    if (m & 1) ok &= add_element_rows<1>(B, r0, len, h.list, m - 1, mh, Kel, slots);
    if (!ok) gfe_raise(err, GFE_DEVERR_SLOT);
    for (int j = lane * 2 - shift; j < len; j += 64) {
      double v[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) v[k] = widen(B[j + k]);
      if (j >= 0 && j + 1 < len) *reinterpret_cast<double2*>(out + j) = make_double2(v[0], v[1]);
      else if (j >= 0) out[j] = v[0];
      else if (len > 0) out[0] = v[1];
    }
    __syncwarp();
  }
}

__global__ void widen_element_matrices(const float* __restrict__ src, size_t n, double* __restrict__ dst) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    dst[i] = (double)src[i / (ND * ND) * kKelF + i % (ND * ND)];
}

// ----------------------------------------------------------------------------------------------
// Consistent tangent of Iron's residual in FP32 (forward-mode dual numbers per Gauss point)
// ----------------------------------------------------------------------------------------------
// Per Gauss point the u-rows of the residual are R(ms,mh) += sum_xi g_ms[xi] P[xi][mh] with
// P = w J_z Z^-1 sigma(Z, p) (Z = dz/dxi, g = reference basis gradients) and the p-rows
// R(ms) += w (J_z - J_x) psi_ms.  The exact derivatives dP/dZ (81 numbers) and dP/dp (9) are
// obtained by 10 forward-mode passes through the same formulas with dual numbers; dJ_z/dZ =
// J_z Z^-T.  The element tangent is then a contraction with the constant basis tables.  This is the derivative that
// Iron's finite-difference Jacobian (src/equations_set_routines.F90:2839-2962) approximates.
template <typename T>
__device__ __forceinline__ T tdet3(const T A[3][3]) {
  return A[0][0] * A[1][1] * A[2][2] + A[0][1] * A[1][2] * A[2][0] + A[0][2] * A[1][0] * A[2][1] -
         A[0][0] * A[2][1] * A[1][2] - A[1][0] * A[0][1] * A[2][2] - A[2][0] * A[1][1] * A[0][2];
}

template <typename T>
__device__ __forceinline__ void tinv3(const T A[3][3], T B[3][3]) {
  const T det = tdet3(A);
  B[0][0] = (A[1][1] * A[2][2] - A[2][1] * A[1][2]) / det;
  B[1][0] = (A[1][2] * A[2][0] - A[2][2] * A[1][0]) / det;
  B[2][0] = (A[1][0] * A[2][1] - A[2][0] * A[1][1]) / det;
  B[0][1] = (A[2][1] * A[0][2] - A[0][1] * A[2][2]) / det;
  B[1][1] = (A[2][2] * A[0][0] - A[0][2] * A[2][0]) / det;
  B[2][1] = (A[2][0] * A[0][1] - A[0][0] * A[2][1]) / det;
  B[0][2] = (A[0][1] * A[1][2] - A[1][1] * A[0][2]) / det;
  B[1][2] = (A[0][2] * A[1][0] - A[1][2] * A[0][0]) / det;
  B[2][2] = (A[0][0] * A[1][1] - A[1][0] * A[0][1]) / det;
}

// forward-mode dual numbers
struct DualF {
  float v, d;
};
__device__ __forceinline__ DualF operator+(DualF a, DualF b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ DualF operator-(DualF a, DualF b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ DualF operator*(DualF a, DualF b) { return {a.v * b.v, a.v * b.d + a.d * b.v}; }
__device__ __forceinline__ DualF operator*(float a, DualF b) { return {a * b.v, a * b.d}; }
__device__ __forceinline__ DualF operator*(DualF a, float b) { return {a.v * b, a.d * b}; }
__device__ __forceinline__ DualF operator/(DualF a, DualF b) {
  const float r = 1.0f / b.v;
  return {a.v * r, (a.d - a.v * r * b.d) * r};
}
__device__ __forceinline__ DualF operator/(DualF a, float b) { return {a.v / b, a.d / b}; }
__device__ __forceinline__ DualF operator+(DualF a, float b) { return {a.v + b, a.d}; }
__device__ __forceinline__ DualF dpowm13(DualF a) {
  const float v = 1.0f / cbrtf(a.v);
  return {v, -v / (3.0f * a.v) * a.d};
}

// P = w Jz Z^-1 sigma(Z, p) of the residual in dual numbers; Jz with its derivative from the caller.
__device__ __forceinline__ void point_P(const DualF (&Z)[3][3], const float A[3][3], float Jx, float w, DualF p,
                                        float c1, float c2, DualF P[3][3], DualF Jz) {
  using T = DualF;
  using R = float;
  T Zi[3][3];
  tinv3(Z, Zi);
  const T J = Jz / Jx;
  const T s = dpowm13(J);
  T Fb[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Fb[i][j] = (Z[i][0] * A[0][j] + Z[i][1] * A[1][j] + Z[i][2] * A[2][j]) * s;
  T C[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) C[i][j] = Fb[0][i] * Fb[0][j] + Fb[1][i] * Fb[1][j] + Fb[2][i] * Fb[2][j];
  const T I1 = C[0][0] + C[1][1] + C[2][2];
  const R t1 = R(-2.0) * c2;
  const T t2 = R(2.0) * (I1 * c2 + c1);
  T Sv[6] = {t1 * C[0][0] + t2, t1 * C[1][1] + t2, t1 * C[2][2] + t2, t1 * C[1][0], t1 * C[2][0], t1 * C[2][1]};
  // sigma_bar = Fb S Fb^T / J (full tensor form of the Voigt push-forward)
  T Sm[3][3] = {{Sv[0], Sv[3], Sv[4]}, {Sv[3], Sv[1], Sv[5]}, {Sv[4], Sv[5], Sv[2]}};
  T FS[3][3], sg[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) FS[i][j] = Fb[i][0] * Sm[0][j] + Fb[i][1] * Sm[1][j] + Fb[i][2] * Sm[2][j];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) sg[i][j] = (FS[i][0] * Fb[j][0] + FS[i][1] * Fb[j][1] + FS[i][2] * Fb[j][2]) / J;
  const T tr3 = (sg[0][0] + sg[1][1] + sg[2][2]) / R(3.0);
#pragma unroll
  for (int i = 0; i < 3; ++i) sg[i][i] = sg[i][i] - tr3 + p;
  const T wj = Jz * w;
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int mh = 0; mh < 3; ++mh) P[k][mh] = wj * (Zi[k][0] * sg[0][mh] + Zi[k][1] * sg[1][mh] + Zi[k][2] * sg[2][mh]);
}

// Gauss-point inputs of the tangent: Z (3x3), the material-frame matrix A, J_x, w, p
template <typename S>
struct GPInT {
  S Z[3][3], A[3][3], Jx, w, p;
};
template <typename S>
__device__ __forceinline__ void gauss_inputs(const TablesT<S>& T, int g, const S* sz, const S* sx, const S* sp,
                                             GPInT<S>& o) {
  S X[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      S a = S(0), b = S(0);
      for (int ns = 0; ns < NQ; ++ns) {
        const S d = T.dphi[g][k][ns];
        a += d * sz[c * NQ + ns];
        b += d * sx[c * NQ + ns];
      }
      o.Z[c][k] = a;
      X[c][k] = b;
    }
  o.Jx = vol_jacobian(X);
  S N[3][3], NX[3][3];
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
  inv3(NX, o.A);
  S p = S(0);
  for (int m = 0; m < NL; ++m) p += T.psi[g][m] * sp[m];
  o.p = p;
  o.w = T.w[g];
}

// J_z = |det Z| and its derivatives for the FP32 dual path, once per Gauss point: the value and the
// signed cofactors (d|det Z| / dZ_ij) in FP64 on the exactly widened entries, rounded to FP32.
// jz[0] = J_z, jz[1 + 3 i + j] = dJ_z/dZ_ij.  The seeds are unit directions, so each seed's
// derivative is one cofactor: forming |det Z| in FP64 dual arithmetic per seed cost about 460 FP64
// operations a Gauss point on GB300's narrow FP64 pipe, this about 30.
__device__ __forceinline__ void jz_seeds(const float (&Zf)[3][3], float jz[10]) {
  double Z[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Z[i][j] = f32_to_f64_exact(Zf[i][j]);
  double cof[3][3];
  cof[0][0] = Z[1][1] * Z[2][2] - Z[1][2] * Z[2][1];
  cof[0][1] = Z[1][2] * Z[2][0] - Z[1][0] * Z[2][2];
  cof[0][2] = Z[1][0] * Z[2][1] - Z[1][1] * Z[2][0];
  cof[1][0] = Z[0][2] * Z[2][1] - Z[0][1] * Z[2][2];
  cof[1][1] = Z[0][0] * Z[2][2] - Z[0][2] * Z[2][0];
  cof[1][2] = Z[0][1] * Z[2][0] - Z[0][0] * Z[2][1];
  cof[2][0] = Z[0][1] * Z[1][2] - Z[0][2] * Z[1][1];
  cof[2][1] = Z[0][2] * Z[1][0] - Z[0][0] * Z[1][2];
  cof[2][2] = Z[0][0] * Z[1][1] - Z[0][1] * Z[1][0];
  const double det = tdet3(Z);
  const double sg = det < 0.0 ? -1.0 : 1.0;
  jz[0] = (float)(sg * det);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) jz[1 + 3 * i + j] = (float)(sg * cof[i][j]);
}

// dP/d(seed) for seed 0..8 = Z[seed/3][seed%3], seed 9 = p.  out[9] = dP[xi][mh] row-major.
// jz: J_z and its seed derivatives from jz_seeds.
__device__ __forceinline__ void point_dP(const GPInT<float>& in, int seed, float c1, float c2, float out[9],
                                         const float jz[10]) {
  DualF Z[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Z[i][j] = {in.Z[i][j], (i * 3 + j == seed) ? 1.0f : 0.0f};
  const DualF p = {in.p, seed == 9 ? 1.0f : 0.0f};
  DualF P[3][3];
  point_P(Z, in.A, in.Jx, in.w, p, c1, c2, P, DualF{jz[0], seed < 9 ? jz[1 + seed] : 0.0f});
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) out[i * 3 + j] = P[i][j].d;
}

// ----------------------------------------------------------------------------------------------
// Element Jacobians: Iron's analytic tangent and the consistent tangent
// ----------------------------------------------------------------------------------------------
// Both are sums over Gauss points of  K(ms mh, ns nh) = g_ms^T D_g^(mh,nh) g_ns  (u-u block) with
// the reference basis gradients g (constant tables) and 3x3 blocks D_g expressed in xi space, plus
// the u-p / p-u blocks.  The work is split in two kernels:
//  * mr_gp_kernel, one thread per (element, Gauss point): kinematics and material tangent, written as
//    D_g (9 blocks x 9), Hv_g (u-p coefficients) and Pv_g (p-u coefficients);
//  * mr_contract_kernel / mr_contract_tc_kernel, one element at a time a CTA: the contraction with the constant
//    table G[(g,xi)][ms] and the u-p / p-u blocks.
// The kernels here serve the FP32 paths (FP32 kinematics with det(F) in FP64, FP32 or TF32 contraction,
// FP64 assembled values).
//
// Iron's analytic tangent (src/finite_elasticity_routines.F90:1016-1274): the spatial blocks
// J_z w (c + sigma) / J_z w c of FINITE_ELASTICITY_GAUSS_ELASTICITY_TENSOR (:649-795) mapped to xi
// space with Z^-1 = dxi/dz (dphi/dz = Z^-T g), only the lower u-u triangle evaluated and mirrored
// to the upper (:1269-1274), p-u = J_z w dphi_ns/dz_nh psi_ms, u-p = J_z w (push(C^-1) dphi_ms)_mh
// psi_ns.  Consistent tangent: D_g^(mh,nh)[xi][zeta] = dP[xi][mh]/dZ[nh][zeta] from the forward-mode
// passes of point_dP, Hv = dP/dp, Pv = w J_z Z^-1.

constexpr int kGPElems = 4;                // elements per CTA of mr_gp_kernel
constexpr uint32_t kTableWaitPolls = 1u << 24;  // bounded wait for the TMA copy of the tables
constexpr int kGPThreads = kGPElems * NG;  // 108
// Gauss-point blocks of an element, floats: D[mh * 3 + nh][g][xi * 3 + zeta] (g padded to 28 with zeros, so that four
// points are nine 16-byte words), Hv[mh][g][xi], Pv[nh][g][xi] (xi padded to 4)
constexpr int kGPBlock = 28 * 9;
constexpr int kGPHv = 9 * kGPBlock;
constexpr int kGPPv = kGPHv + 3 * NG * 4;
constexpr int kGPItem = kGPPv + 3 * NG * 4;  // 2916: a 16-byte multiple (TMA)
static_assert(kGPBlock % 4 == 0 && kGPItem % 4 == 0, "TMA bulk copies");

struct GPShared {
  alignas(16) float out[2][kGPElems][3 * kGPBlock];  // staging of the blocks: three (mh, nh) pairs, or Hv and Pv
  float x[kGPElems][81], z[kGPElems][81], p[kGPElems][8];
};
static_assert(kGPItem - kGPHv <= 3 * kGPBlock, "Hv and Pv fit one stage");

// One thread per (element, Gauss point), blocks at out[item * kGPItem].  They leave through shared memory, the three
// blocks of one nh at a time, by TMA bulk copies: a thread's own stores are 4 bytes 36 apart, a sector each (32^3
// elements: 498 -> 419 us; now bound by the FP32 instructions of the ten passes at 16 warps an SM; three seeds a pass
// take 235 registers, 548 us).  Element data
// rounded to FP32 once per
// node when staged, the volume Jacobians det(Z), det(X) still evaluated in FP64 from the exactly widened
// gradients; for the consistent tangent (EXACT) the forward-mode passes run in FP32 dual numbers, with
// J_z and its derivatives formed in FP64 once a point (jz_seeds).
template <bool EXACT>
__global__ void __launch_bounds__(kGPThreads, 4)
mr_gp_kernel(const int32_t* __restrict__ elems, int32_t count, const int32_t* __restrict__ eq2,
             const int32_t* __restrict__ elin, int32_t nq2, const double* __restrict__ xg,
             const double* __restrict__ dep, const double* __restrict__ cpar, const TablesF* __restrict__ Tg,
             float* __restrict__ out, unsigned* err) {
  extern __shared__ __align__(16) double smem_d[];
  unsigned char* sbase = reinterpret_cast<unsigned char*>(smem_d);
  TablesF& T = *reinterpret_cast<TablesF*>(sbase);
  GPShared& S = *reinterpret_cast<GPShared*>(sbase + sizeof(TablesF));
  uint64_t* tbar = reinterpret_cast<uint64_t*>(sbase + sizeof(TablesF) + sizeof(GPShared));
  // the basis tables arrive by one TMA bulk copy while the threads gather the element data
  if (threadIdx.x == 0) {
    tc::mbar_init(tbar, 1);
    tc::mbar_arrive_expect_tx(tbar, (uint32_t)sizeof(TablesF));
    tc::bulk_copy_g2s(&T, Tg, (uint32_t)sizeof(TablesF), tbar);
  }
  const int le = threadIdx.x / NG, g = threadIdx.x % NG;
  const int item = blockIdx.x * kGPElems + le;
  // cooperative load of the CTA's elements
  for (int t = threadIdx.x; t < kGPElems * NQ; t += blockDim.x) {
    const int l = t / NQ, i = t % NQ, it = blockIdx.x * kGPElems + l;
    if (it >= count) continue;
    const int e = __ldg(elems + it);
    const int n = __ldg(eq2 + (size_t)e * NQ + i);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      S.x[l][c * NQ + i] = (float)__ldg(xg + (size_t)c * nq2 + n);
      S.z[l][c * NQ + i] = (float)dep[(size_t)c * nq2 + n];
    }
  }
  for (int t = threadIdx.x; t < kGPElems * NL; t += blockDim.x) {
    const int l = t / NL, i = t % NL, it = blockIdx.x * kGPElems + l;
    if (it >= count) continue;
    const int e = __ldg(elems + it);
    S.p[l][i] = (float)dep[(size_t)3 * nq2 + __ldg(elin + (size_t)e * NL + i)];
  }
  __syncthreads();
  // every thread waits for the tables (so none exits while the copy is in flight); bounded
  if (!tc::mbar_wait(tbar, 0, kTableWaitPolls)) {
    gfe_raise(err, GFE_DEVERR_TIMEOUT);
    tc::mbar_wait(tbar, 0, kTableWaitPolls);
    return;
  }
  const bool live = item < count;
  const int n_live = min(kGPElems, count - (int)blockIdx.x * kGPElems);
  // stage nh of the element's blocks, o[mh * kGPBlock + g * 9 + xi * 3 + zeta], or (nh = 3) Hv and Pv; then the
  // copies of one stage run while the next is formed in the other half
  auto stage = [&](int nh) { return S.out[nh & 1][le] + (nh < 3 ? g * 9 : g * 4); };
  auto begin_stage = [&](int nh) {
    if (nh >= 2) {
      if (threadIdx.x == 0) tc::bulk_wait_read<1>();
      __syncthreads();
    }
  };
  auto end_stage = [&](int nh) {
    if (nh < 3 && g == NG - 1)
      for (int mh = 0; mh < 3; ++mh)
        for (int k = 0; k < 9; ++k) S.out[nh & 1][le][mh * kGPBlock + NG * 9 + k] = 0.0f;
    tc::fence_proxy_async();
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int l = 0; l < n_live; ++l) {
        float* dst = out + ((size_t)blockIdx.x * kGPElems + l) * kGPItem;
        if (nh < 3) {
          for (int mh = 0; mh < 3; ++mh)
            tc::bulk_copy_s2g(dst + (mh * 3 + nh) * kGPBlock, S.out[nh & 1][l] + mh * kGPBlock, kGPBlock * 4);
        } else {
          tc::bulk_copy_s2g(dst + kGPHv, S.out[nh & 1][l], (kGPItem - kGPHv) * 4);
        }
      }
      tc::bulk_commit();
    }
  };
  if constexpr (!EXACT) {
    const float c1 = (float)cpar[0], c2 = (float)cpar[1];
    GPT<float> q;
    float sub[6][9], hyd[9], jgw = 0.0f;
    if (live) {
      if (!gauss_point(T, g, S.z[le], S.x[le], S.p[le], q)) gfe_raise(err, GFE_DEVERR_JACOBIAN);
      iron_point_tensors(q, c1, c2, sub, hyd, jgw);
    }
    // blocks to xi space: Dxi = Zi sub Zi^T (Zi = dxi/dz); upper blocks as transposes of the lower
#pragma unroll
    for (int nh = 0; nh < 3; ++nh) {
      begin_stage(nh);
      float* o = stage(nh);
      if (live) {
#pragma unroll
        for (int mh = 0; mh < 3; ++mh) {
          const int blk = mh == nh ? mh : (mh > nh ? 3 + (mh == 1 ? 0 : (nh == 0 ? 1 : 2))
                                                   : 3 + (nh == 1 ? 0 : (mh == 0 ? 1 : 2)));
          const bool tr = mh < nh;
          float W[3][3];
#pragma unroll
          for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int z = 0; z < 3; ++z) {
              float s = float(0);
#pragma unroll
              for (int j = 0; j < 3; ++j) s += (tr ? sub[blk][j * 3 + i] : sub[blk][i * 3 + j]) * q.Zi[z][j];
              W[i][z] = s;  // (sub Zi^T)[i][zeta]
            }
#pragma unroll
          for (int xi = 0; xi < 3; ++xi)
#pragma unroll
            for (int z = 0; z < 3; ++z)
              o[mh * kGPBlock + xi * 3 + z] =
                  (float)(q.Zi[xi][0] * W[0][z] + q.Zi[xi][1] * W[1][z] + q.Zi[xi][2] * W[2][z]);
        }
      }
      end_stage(nh);
    }
    begin_stage(3);
    float* o = stage(3);
    if (live) {
#pragma unroll
      for (int xi = 0; xi < 3; ++xi)
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          o[m * NG * 4 + xi] = (float)(q.Zi[xi][0] * hyd[m * 3 + 0] + q.Zi[xi][1] * hyd[m * 3 + 1] +
                                       q.Zi[xi][2] * hyd[m * 3 + 2]);
          o[kGPPv - kGPHv + m * NG * 4 + xi] = (float)(jgw * q.Zi[xi][m]);
        }
    }
    end_stage(3);
  } else {
    const float c1 = (float)cpar[0], c2 = (float)cpar[1];
    GPInT<float> in;
    float jz[10];
    if (live) {
      gauss_inputs(T, g, S.z[le], S.x[le], S.p[le], in);
      jz_seeds(in.Z, jz);
    }
    for (int nh = 0; nh < 4; ++nh) {
      begin_stage(nh);
      float* o = stage(nh);
      if (live) {
        for (int z = 0; z < (nh < 3 ? 3 : 1); ++z) {
          float d[9];
          point_dP(in, nh * 3 + z, c1, c2, d, jz);
#pragma unroll
          for (int xi = 0; xi < 3; ++xi)
#pragma unroll
            for (int mh = 0; mh < 3; ++mh) {
              if (nh < 3) o[mh * kGPBlock + xi * 3 + z] = d[xi * 3 + mh];
              else o[mh * NG * 4 + xi] = d[xi * 3 + mh];
            }
        }
        if (nh == 3) {
          float Zi[3][3];
          const float dz = inv3(in.Z, Zi);
          if (!(dz > float(0)) || !isfinite(dz)) gfe_raise(err, GFE_DEVERR_JACOBIAN);
#pragma unroll
          for (int xi = 0; xi < 3; ++xi)
#pragma unroll
            for (int m = 0; m < 3; ++m) o[kGPPv - kGPHv + m * NG * 4 + xi] = (float)(in.w * jz[0] * Zi[xi][m]);
        }
      }
      end_stage(nh);
    }
  }
  if (threadIdx.x == 0) tc::bulk_wait_read<0>();  // the stages may be gone once this thread exits
}

__device__ __forceinline__ void load4(const float* p, float* v) {
  const float4 q = *reinterpret_cast<const float4*>(p);
  v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}

// u-p / p-u blocks of one element into its matrix K: a warp has component h, its lanes ms; both are 27-term sums with
// the pressure basis.
template <typename Wait>
__device__ __forceinline__ void up_blocks(int h, const float* Dg, const float (*G)[28], const float (*psi)[NL], float* K,
                                          Wait wait) {
  const int lane = threadIdx.x & 31, ms = min(lane, 26), r = h * 27 + ms;
  const float4* H4 = reinterpret_cast<const float4*>(Dg + kGPHv) + h * NG;
  const float4* P4 = reinterpret_cast<const float4*>(Dg + kGPPv) + h * NG;
  float up[NL], pu[NL];
#pragma unroll
  for (int b = 0; b < NL; ++b) up[b] = pu[b] = 0.0f;
#pragma unroll 3
  for (int g = 0; g < NG; ++g) {
    const float4 H = H4[g], P = P4[g];
    const float g0 = G[g * 3][ms], g1 = G[g * 3 + 1][ms], g2 = G[g * 3 + 2][ms];
    const float hg = g0 * H.x + g1 * H.y + g2 * H.z;
    const float pg = g0 * P.x + g1 * P.y + g2 * P.z;
    float q[NL];
    load4(&psi[g][0], q);
    load4(&psi[g][4], q + 4);
#pragma unroll
    for (int b = 0; b < NL; ++b) {
      up[b] += hg * q[b];
      pu[b] += q[b] * pg;
    }
  }
  if (!wait()) return;
  if (lane < 27) {
#pragma unroll
    for (int b = 0; b < NL; ++b) {
      K[r * ND + 81 + b] = up[b];
      K[(81 + b) * ND + r] = pu[b];
    }
  }
}

// CUDA-core form of the product of the tensor-core kernel below,
//   C[(mh,nh,ms)][ns] = sum_{(g,zeta)} A[(mh,nh,ms)][(g,zeta)] G[(g,zeta)][ns],
//   A[(mh,nh,ms)][(g,zeta)] = sum_xi G[(g,xi)][ms] D_g[(mh,nh)][xi][zeta],
// 243 x 81 by 81 x 27.  A thread owns a row of C for two elements: it forms A's entries in registers as it goes and
// takes a row of G, the same for all threads, by 16-byte broadcasts, 54 FMAs for seven.  Bound by the issue of the FMAs
// (about 6,100 cycles an element and SM).  With A in shared memory and a 4 x 4 tile a thread, two vector loads for
// 16 FMAs, 32^3 elements took 2,869 us, now 1,240.
constexpr int kCThreads = 256;

struct ContractShared {
  alignas(16) float G[81][28];          // G[(g,xi)][ms]; column 27 zero
  alignas(16) float psi[NG][NL];        // pressure basis at the Gauss points
  alignas(16) float Dg[2][kGPItem];     // the two elements' Gauss-point blocks
  alignas(16) float K[2][kKelF];        // and matrices
};

// Element matrices of `count` elements into Kel[e * kKelF] (element number e = elems[item]).
template <bool EXACT>
__global__ void __launch_bounds__(kCThreads, 2)
mr_contract_kernel(const int32_t* __restrict__ elems, int32_t count, const Tables* __restrict__ Tg,
                   const float* __restrict__ gp, float* __restrict__ Kel) {
  extern __shared__ __align__(16) unsigned char craw[];
  ContractShared& S = *reinterpret_cast<ContractShared*>(craw);
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int t = tid; t < 81 * 28; t += kCThreads) {
    const int k = t / 28, ms = t % 28;
    S.G[k][ms] = ms < 27 ? (float)Tg->dphi[k / 3][k % 3][ms] : 0.0f;
  }
  for (int t = tid; t < NG * NL; t += kCThreads) S.psi[t / NL][t % NL] = (float)Tg->psi[t / NL][t % NL];
  // the zero p-p blocks and the padding behind the matrices are never written again
  for (int t = tid; t < 2 * NL * NL; t += kCThreads) S.K[t / 64][(81 + t % 64 / NL) * ND + 81 + t % NL] = 0.0f;
  if (tid < 2 * (kKelF - ND * ND)) S.K[tid & 1][ND * ND + (tid >> 1)] = 0.0f;
  const int row = tid, pair = min(row / 27, 8), ms = row % 27, mh = pair / 3, nh = pair % 3, r = mh * 27 + ms;
  for (int item = blockIdx.x * 2; item < count; item += gridDim.x * 2) {
    const int n_live = min(2, count - item);
    if (tid == 0) tc::bulk_wait_read<0>();  // the matrices of the round before have been read
    __syncthreads();
    const float4* src = reinterpret_cast<const float4*>(gp + (size_t)item * kGPItem);
    float4* dst = reinterpret_cast<float4*>(&S.Dg[0][0]);
    for (int t = tid; t < n_live * kGPItem / 4; t += kCThreads) dst[t] = __ldg(src + t);
    __syncthreads();
    if (row < 243) {
      float acc[2][27];
#pragma unroll
      for (int n = 0; n < 27; ++n) acc[0][n] = acc[1][n] = 0.0f;
#pragma unroll 1
      for (int g = 0; g < NG; ++g) {
        const float g0 = S.G[g * 3][ms], g1 = S.G[g * 3 + 1][ms], g2 = S.G[g * 3 + 2][ms];
        float a[2][3];
#pragma unroll
        for (int l = 0; l < 2; ++l) {
          const float* D = S.Dg[l] + pair * kGPBlock + g * 9;
#pragma unroll
          for (int z = 0; z < 3; ++z) a[l][z] = g0 * D[z] + g1 * D[3 + z] + g2 * D[6 + z];
        }
#pragma unroll
        for (int z = 0; z < 3; ++z) {
          float b[28];
#pragma unroll
          for (int q = 0; q < 7; ++q) load4(&S.G[g * 3 + z][4 * q], b + 4 * q);
#pragma unroll
          for (int n = 0; n < 27; ++n) {
            acc[0][n] += a[0][z] * b[n];
            acc[1][n] += a[1][z] * b[n];
          }
        }
      }
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        float* Kr = S.K[l] + r * ND + nh * 27;
        float* Kc = S.K[l] + nh * 27 * ND + r;
#pragma unroll
        for (int n = 0; n < 27; ++n) {
          // Iron mirrors the lower triangle into the upper one unless EXACT
          if (EXACT || r >= nh * 27 + n) Kr[n] = acc[l][n];
          if (!EXACT && r >= nh * 27 + n) Kc[n * ND] = acc[l][n];
        }
      }
    }
    if (warp < 6) up_blocks(warp % 3, S.Dg[warp / 3], S.G, S.psi, S.K[warp / 3], [] { return true; });
    tc::fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      for (int l = 0; l < n_live; ++l)
        tc::bulk_copy_s2g(Kel + (size_t)__ldg(elems + item + l) * kKelF, S.K[l], kKelF * (uint32_t)sizeof(float));
      tc::bulk_commit();
    }
  }
  if (tid == 0) tc::bulk_wait_read<0>();  // shared memory may be gone once this thread exits
}

// ---------------------------------------------------------------------------------------------
// Tensor-core (tcgen05, TF32) basis-gradient contraction of the element Jacobian
// ---------------------------------------------------------------------------------------------
// For every (mh, nh) displacement-component pair the u-u block is
//   K[(ms,mh),(ns,nh)] = sum_{g,zeta} A[(mh,nh,ms)][(g,zeta)] G[(g,zeta)][ns],
//   A[(mh,nh,ms)][(g,zeta)] = sum_xi G[(g,xi)][ms] D_g[(mh,nh)][xi][zeta],
// i.e. one 243 x 81 by 81 x 27 product per element, as two M = 128 halves of tcgen05.mma kind::tf32 (N = 32, K = 88
// in 11 steps of 8).  With SPLIT3 each operand is split into a TF32 head and a TF32 tail and the three products
// hi*hi + lo*hi + hi*lo recover about FP32 accuracy; without it the contraction is plain TF32 (about 1e-3
// relative).
//
// With A formed in shared memory (one CTA an SM, every phase behind the other) this took 2,073 us for 32^3 elements:
// 5,600 wavefronts of shared memory an element for forming A, 2,600 cycles for the MMAs' operand reads and a single
// thread's descriptor arithmetic.  Now (665 us) a thread forms a part of a row of A in registers (D by 16-byte
// broadcasts, G without bank conflicts) and stores it to tensor memory, from which the MMAs take it; only the constant
// G^T stays in shared memory, and the finished matrix leaves by one bulk copy.  The MMAs bound it: each takes 48
// cycles for any N up to 64, 66 of them 3,200 cycles an element, and stores to tensor memory wait while MMAs of
// either CTA run.  Hence two CTAs an SM that alternate, and large stores.  Slower: forming one K chunk while the
// other is multiplied (801 us: the stores wait), one CTA that keeps a half of A in registers (952 us).  The head of
// the split is rounded on the integer pipe (706 us with two conversions an entry).
constexpr int kTCThreads = 384;
constexpr int kTCForm = 8, kTCUp = 3;  // warps 0 .. 7 (two a tensor-memory quadrant), 8 .. 10; 11 copies and MMAs
constexpr int kTK = 88;                        // K = 27 Gauss points x 3, padded to 11 steps of 8
constexpr int kTKC = kTK / 4;                  // core-matrix columns along K (4 TF32 = 16 bytes)
constexpr int kTBBytes = 4 * kTKC * 128;       // the N = 32 operand
constexpr uint32_t kTLbo = 128, kTSbo = kTKC * 128;
// tensor memory: a half of A, its K columns as 24 heads, 24 tails, 24 heads, ..., 16 heads, 16 tails; the two halves'
// products
constexpr uint32_t kTCols = 256;
constexpr uint32_t kTAccCol = 2 * kTK;
__host__ __device__ constexpr uint32_t tc_a_col(int step) { return (uint32_t)(step / 3 * 48 + step % 3 * 8); }
__host__ __device__ constexpr uint32_t tc_a_tail(int step) { return step < 9 ? 24u : 16u; }
constexpr long long kTWaitCycles = 2000000000; // bounded waits: about a second

struct __align__(128) TCShared {
  unsigned char B[2][kTBBytes];  // G head, tail: B[ns][(g,zeta)]
  float G[84][28];               // G[(g,xi)][ms]; column 27 and rows 81 .. 83 zero
  alignas(16) float psi[NG][NL];
  alignas(16) float Dg[2][kGPItem];  // Gauss-point blocks of the current and the next element (TMA)
  alignas(16) float K[kKelF];    // the element matrix
  uint64_t afull, acc;           // a half of A formed / multiplied
  uint64_t dfull[2];             // bulk copies into Dg[0], Dg[1]
  uint64_t kfull, kempty;        // K written by the other warps / copied out
  uint32_t tmem;
  int undrained;
};

// byte offset of element (row, k) in a no-swizzle K-major operand with kTKC core columns
__device__ __forceinline__ uint32_t tc_offset(int row, int k) {
  return (uint32_t)((((row >> 3) * kTKC + (k >> 2)) * 8 + (row & 7)) * 16 + (k & 3) * 4);
}

// Warp: waits for the phase of parity `parity`; false after about a second.
__device__ __forceinline__ bool tc_wait(uint64_t* mbar, uint32_t parity, unsigned* err) {
  bool ok = tc::mbar_wait(mbar, parity, 16);
  if (!ok) {
    const long long t0 = clock64();
    while (!(ok = tc::mbar_wait(mbar, parity, 16)) && clock64() - t0 < kTWaitCycles) {
    }
  }
  ok = __all_sync(0xffffffffu, ok);
  if (!ok) gfe_raise(err, GFE_DEVERR_TIMEOUT);
  return ok;
}

template <bool EXACT, bool SPLIT3>
__global__ void __launch_bounds__(kTCThreads, 2)
mr_contract_tc_kernel(const int32_t* __restrict__ elems, int32_t count, const Tables* __restrict__ Tg,
                      const float* __restrict__ gp, float* __restrict__ Kel, unsigned* err) {
  extern __shared__ __align__(1024) unsigned char traw[];
  TCShared& S = *reinterpret_cast<TCShared*>(traw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr uint32_t kDgBytes = kGPItem * sizeof(float);
  // constant operands: G (FP32, for forming A) and B = G^T split into TF32 head / tail
  for (int t = tid; t < 84 * 28; t += kTCThreads) {
    const int k = t / 28, ms = t % 28;
    S.G[k][ms] = ms < 27 && k < 81 ? (float)Tg->dphi[k / 3][k % 3][ms] : 0.0f;
  }
  for (int t = tid; t < NG * NL; t += kTCThreads) S.psi[t / NL][t % NL] = (float)Tg->psi[t / NL][t % NL];
  for (int t = tid; t < 32 * kTK; t += kTCThreads) {
    const int n = t / kTK, k = t % kTK;
    const float v = (n < 27 && k < 81) ? (float)Tg->dphi[k / 3][k % 3][n] : 0.0f;
    const float hi = tc::to_tf32(v);
    *reinterpret_cast<float*>(S.B[0] + tc_offset(n, k)) = hi;
    *reinterpret_cast<float*>(S.B[1] + tc_offset(n, k)) = tc::to_tf32(v - hi);
  }
  // the zero p-p block and the padding behind the matrix are never written again
  for (int t = tid; t < NL * NL; t += kTCThreads) S.K[(81 + t / NL) * ND + 81 + t % NL] = 0.0f;
  if (tid < kKelF - ND * ND) S.K[ND * ND + tid] = 0.0f;
  if (warp == 0) tc::tmem_alloc(&S.tmem, kTCols);
  if (tid == 0) {
    tc::mbar_init(&S.afull, kTCForm);
    tc::mbar_init(&S.acc, 1);
    tc::mbar_init(&S.dfull[0], 1);
    tc::mbar_init(&S.dfull[1], 1);
    tc::mbar_init(&S.kfull, kTCForm + kTCUp);
    tc::mbar_init(&S.kempty, 1);
    S.undrained = 0;
  }
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, S.tmem, 0);

  if (warp < kTCForm) {
    // rows half * 128 + 32 warp + lane of A, formed four Gauss points (12 columns) at a time
    const uint32_t quad = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int part = warp >> 2;  // columns 0 .. 47, or 48 .. 87
    // head and tail of the 12 columns of Gauss points 4 gg .. 4 gg + 3
    auto form12 = [&](const float4* D4, const float* Gm, int gg, float* hi, float* lo) {
      float d[36];
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const float4 t = D4[gg * 9 + q];
        d[4 * q] = t.x;
        d[4 * q + 1] = t.y;
        d[4 * q + 2] = t.z;
        d[4 * q + 3] = t.w;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float* Gg = Gm + (gg * 4 + u) * 3 * 28;
        const float g0 = Gg[0], g1 = Gg[28], g2 = Gg[56];
#pragma unroll
        for (int z = 0; z < 3; ++z) {
          const float v = g0 * d[u * 9 + z] + g1 * d[u * 9 + 3 + z] + g2 * d[u * 9 + 6 + z];
          hi[u * 3 + z] = SPLIT3 ? tc::to_tf32_number(v) : tc::to_tf32(v);
          if (SPLIT3) lo[u * 3 + z] = tc::to_tf32(v - hi[u * 3 + z]);
        }
      }
    };
    // A store to tensor memory waits for the MMA in flight, so it takes 24 columns (head and tail) at once: with
    // 12 columns in four stores, forming took twice as long
    auto form = [&](const float* Dg, int half) {
      const int row = half * 128 + (warp & 3) * 32 + lane, pair = min(row / 27, 8), ms = row % 27;
      const float4* D4 = reinterpret_cast<const float4*>(Dg + pair * kGPBlock) + part * 36;
      const float* Gm = &S.G[part * 48][ms];
      const uint32_t base = quad + (uint32_t)(part * 96);
      auto form24 = [&](int h) {
        float v[48];  // 24 heads, 24 tails
        form12(D4, Gm, h * 2, v, v + 24);
        form12(D4, Gm, h * 2 + 1, v + 12, v + 36);
        if (SPLIT3) {
          tc::tmem_st_32(base + h * 48, v);
          tc::tmem_st_16(base + h * 48 + 32, v + 32);
        } else {
          tc::tmem_st_16(base + h * 48, v);
          tc::tmem_st_8(base + h * 48 + 16, v + 16);
        }
      };
      form24(0);
      if (part == 0) {
        form24(1);
      } else {
        float v[32];  // 12 heads, 4 zeros, 12 tails, 4 zeros
        form12(D4, Gm, 2, v, v + 16);
#pragma unroll
        for (int k = 12; k < 16; ++k) v[k] = v[16 + k] = 0.0f;
        if (SPLIT3) tc::tmem_st_32(base + 48, v);
        else tc::tmem_st_16(base + 48, v);
      }
      tc::tmem_wait_st();
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&S.afull);
    };
    // the products of a half into the element matrix
    auto read_back = [&](int half) {  // columns 0 .. 15, or 16 .. 26
      float v[16];
      tc::fence_after_sync();
      tc::tmem_ld_32x16(quad + kTAccCol + (uint32_t)(half * 32 + part * 16), v);
      const int row = half * 128 + (warp & 3) * 32 + lane, pair = min(row / 27, 8), ms = row % 27;
      if (row >= 243) return;
      const int mh = pair / 3, nh = pair % 3, r = mh * 27 + ms, n0 = part * 16;
      float* Kr = S.K + r * ND + nh * 27 + n0;
      float* Kc = S.K + (nh * 27 + n0) * ND + r;
#pragma unroll
      for (int n = 0; n < 16; ++n) {
        if (n >= 11 && part) break;
        // Iron mirrors the lower triangle into the upper one unless EXACT
        if (EXACT || r >= nh * 27 + n0 + n) Kr[n] = v[n];
        if (!EXACT && r >= nh * 27 + n0 + n) Kc[n * ND] = v[n];
      }
    };
    for (int i = 0, item = blockIdx.x; item < count; ++i, item += gridDim.x) {
      if (!tc_wait(&S.dfull[i & 1], (uint32_t)(i >> 1) & 1u, err)) break;
      form(S.Dg[i & 1], 0);
      if (!tc_wait(&S.acc, 0u, err) || (i > 0 && !tc_wait(&S.kempty, (uint32_t)(i - 1) & 1u, err))) break;
      read_back(0);
      form(S.Dg[i & 1], 1);
      if (!tc_wait(&S.acc, 1u, err)) break;
      read_back(1);
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&S.kfull);
    }
  } else if (warp < kTCForm + kTCUp) {
    // u-p / p-u blocks
    for (int i = 0, item = blockIdx.x; item < count; ++i, item += gridDim.x) {
      if (!tc_wait(&S.dfull[i & 1], (uint32_t)(i >> 1) & 1u, err)) break;
      bool ok = true;
      up_blocks(warp - kTCForm, S.Dg[i & 1], S.G, S.psi, S.K,
                [&] { return ok = i == 0 || tc_wait(&S.kempty, (uint32_t)(i - 1) & 1u, err); });
      if (!ok) break;
      tc::fence_proxy_async();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&S.kfull);
    }
  } else if (lane == 0) {
    // the next elements' blocks in, the MMAs as the halves of A come, the matrices out
    constexpr uint32_t idesc = tc::idesc_tf32(128, 32);
    const uint64_t b_hi = tc::smem_desc(tc::smem_u32(S.B[0]), kTLbo, kTSbo);
    const uint64_t b_lo = tc::smem_desc(tc::smem_u32(S.B[1]), kTLbo, kTSbo);
    auto load = [&](int i, int item) {
      tc::mbar_arrive_expect_tx(&S.dfull[i & 1], kDgBytes);
      tc::bulk_copy_g2s(S.Dg[i & 1], gp + (size_t)item * kGPItem, kDgBytes, &S.dfull[i & 1]);
    };
    auto wait = [&](uint64_t* mbar, uint32_t parity) {
      const long long t0 = clock64();
      while (!tc::mbar_wait(mbar, parity, 16))
        if (clock64() - t0 > kTWaitCycles) {
          gfe_raise(err, GFE_DEVERR_TIMEOUT);
          return false;
        }
      return true;
    };
    const int step = (int)gridDim.x;
    for (int k = 0; k < 2; ++k)
      if ((int)blockIdx.x + k * step < count) load(k, blockIdx.x + k * step);
    bool ok = true;
    int i = 0;
    for (int item = blockIdx.x; item < count; ++i, item += step) {
      for (int half = 0; half < 2; ++half) {
        if (!(ok = wait(&S.afull, (uint32_t)half))) break;
        tc::fence_after_sync();
        const uint32_t d = tmem + kTAccCol + (uint32_t)(half * 32);
#pragma unroll
        for (int s = 0; s < kTK / 8; ++s) {
          const uint32_t a = tmem + tc_a_col(s);
          tc::mma_tf32_ts(d, a, b_hi + s * 16, idesc, s > 0 ? 1u : 0u);  // a step is 256 bytes: 16 in the descriptor
          if (SPLIT3) {
            tc::mma_tf32_ts(d, a + tc_a_tail(s), b_hi + s * 16, idesc, 1u);
            tc::mma_tf32_ts(d, a, b_lo + s * 16, idesc, 1u);
          }
        }
        tc::commit(&S.acc);
      }
      // every warp is done with this element (and the MMAs are, as their products have been read): its matrix goes
      // out and its blocks' buffer is free
      if (!ok || !(ok = wait(&S.kfull, (uint32_t)i & 1u))) break;
      tc::fence_proxy_async();
      tc::bulk_copy_s2g(Kel + (size_t)__ldg(elems + item) * kKelF, S.K, kKelF * (uint32_t)sizeof(float));
      tc::bulk_commit();
      if (item + 2 * step < count) load(i + 2, item + 2 * step);
      tc::bulk_wait_read<0>();
      tc::mbar_arrive(&S.kempty);
    }
    if (!ok) {
      // MMAs may still write tensor memory: it stays allocated.  No copy may still be landing in this CTA's shared
      // memory when it exits
      S.undrained = 1;
      for (int k = i; k < i + 2; ++k)
        if ((int)blockIdx.x + k * step < count) wait(&S.dfull[k & 1], (uint32_t)(k >> 1) & 1u);
    }
  }
  __syncwarp();
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0 && !S.undrained) tc::tmem_dealloc(tmem, kTCols);
}

int check_mesh(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin, const double* xg,
               const char* fn) {
  if (n_elem < 0 || nq2 <= 0 || nlin <= 0 || (n_elem > 0 && (!eq2 || !elin || !xg)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid mesh arguments", fn);
  return GFE_OK;
}

int set_smem(const void* kernel, size_t bytes) {
  GFE_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return GFE_OK;
}

}  // namespace

extern "C" int gfe_mr_slot_map(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2,
                               const int32_t* color_elems, const int32_t* row_ptr, const int32_t* col_idx,
                               int32_t* slots, void* stream) {
  const char* fn = "gfe_mr_slot_map";
  if (n_elem < 0 || !eq2 || !elin || !color_elems || !row_ptr || !col_idx || !slots)
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid arguments", fn);
  if (n_elem == 0) return GFE_OK;
  cudaStream_t s = gfe::as_stream(stream);
  mr_slot_kernel<<<16 * gfe::sm_count(), 256, 0, s>>>(color_elems, n_elem, eq2, elin, nq2, row_ptr, col_idx, slots);
  GFE_LAUNCH_CHECK(fn);
  return GFE_OK;
}

namespace {

// Element Jacobians of one problem (mode 0: Iron's analytic tangent, 1: consistent tangent), in the
// contraction precision `precision`.  Elements in chunks of at most kElemChunk: the Gauss-point
// kernel fills a scratch array, the contraction kernel turns it into element matrices Kel (all
// elements; FP64 for GFE_FP64, else FP32); then the row gather assembles the CSR values (when
// `values`), and K_out receives the element matrices in FP64 (when given).
constexpr int kElemChunk = 1 << 16;

template <bool EXACT, bool SPLIT3>
void launch_contract_tc(int grid, cudaStream_t s, const int32_t* elems, int cnt, const Tables* T, const float* gp,
                        float* Kel, unsigned* err) {
  mr_contract_tc_kernel<EXACT, SPLIT3><<<grid, kTCThreads, sizeof(TCShared), s>>>(elems, cnt, T, gp, Kel, err);
}

// Node incidence scratch (counts, then lists) and the row gather into `values`.
template <typename TS>
int gather_rows(int32_t n_elem, const int32_t* elems, const int32_t* eq2, const int32_t* elin, int32_t nq2,
                int32_t nlin, const TS* Kel, const int32_t* slots, const int32_t* row_ptr, double* values,
                cudaStream_t s, unsigned* err) {
  const int32_t n_nodes = nq2 + nlin;
  int32_t* inc = nullptr;
  const size_t words = (size_t)n_nodes * (1 + kMaxInc);
  int rc = gfe::scratch_alloc((void**)&inc, sizeof(int32_t) * words, s, "node incidence");
  if (rc) return rc;
  int32_t* cnt = inc;
  int32_t* list = inc + n_nodes;
  cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (size_t)n_nodes, s);
  if (e != cudaSuccess) {
    gfe::scratch_free(inc, s);
    return gfe::set_error(GFE_ERR_CUDA, "node incidence: %s", cudaGetErrorString(e));
  }
  const int sms = gfe::sm_count();
  mr_incidence_fill<<<8 * sms, 256, 0, s>>>(elems, n_elem, eq2, elin, nq2, cnt, list, err);
  mr_incidence_sort<<<(n_nodes + 255) / 256, 256, 0, s>>>(n_nodes, cnt, list);
  const long long rows = 3ll * nq2 + nlin;
  const int grid = (int)std::min<long long>((rows + kRowWarps - 1) / kRowWarps, 16ll * sms);
  mr_row_gather_kernel<TS><<<grid, kRowWarps * 32, 0, s>>>(nq2, nlin, cnt, list, Kel, slots, row_ptr, values,
                                                          err);
  gfe::scratch_free(inc, s);
  return GFE_OK;
}

// FP64: mr_jac64.cu forms the element matrices, straight into K_out when it is given.
int jacobian_f64(int mode, int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin,
                 const double* xg, const int32_t* elems, const double* dep, const double* cpar, const int32_t* slots,
                 const int32_t* row_ptr, double* values, double* K_out, cudaStream_t s, const char* fn) {
  if (n_elem == 0) return GFE_OK;
  int rc;
  double* Kel = K_out;
  if (!K_out && (rc = gfe::scratch_alloc((void**)&Kel, sizeof(double) * (size_t)n_elem * ND * ND, s, "element matrices")))
    return rc;
  unsigned* err = gfe::device_error_word();
  void* prof = gfe::stage_begin(GFE_STAGE_MR_JACOBIAN, s);
  int launches = 0;
  rc = mr64::element_matrices(mode != 0, n_elem, elems, eq2, elin, nq2, xg, dep, cpar, Kel, s, err, &launches);
  if (!rc && values) rc = gather_rows<double>(n_elem, elems, eq2, elin, nq2, nlin, Kel, slots, row_ptr, values, s, err);
  gfe::stage_end(GFE_STAGE_MR_JACOBIAN, prof, s, launches + (values ? 3 : 0));
  if (!K_out) gfe::scratch_free(Kel, s);
  if (rc) return rc;
  GFE_LAUNCH_CHECK(fn);
  return GFE_OK;
}

// FP32 kinematics and contraction (tc_mode 0: CUDA cores, else the tensor cores).
int jacobian_f32(int mode, int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin,
                 const double* xg, const int32_t* elems, const double* dep, const double* cpar, const int32_t* slots,
                 const int32_t* row_ptr, double* values, double* K_out, cudaStream_t s, const char* fn, int tc_mode) {
  const Tables* T = nullptr;
  int rc = device_tables(&T);
  if (rc) return rc;
  const TablesF* TK = nullptr;
  if ((rc = device_tables_f(&TK))) return rc;
  if (n_elem == 0) return GFE_OK;
  const size_t gsm_k = sizeof(TablesF) + sizeof(GPShared) + 16;  // + the tables' mbarrier
  const size_t csm = sizeof(ContractShared);
  const void* gk = mode == 0 ? (const void*)mr_gp_kernel<false> : (const void*)mr_gp_kernel<true>;
  const void* ck = mode == 0 ? (const void*)mr_contract_kernel<false> : (const void*)mr_contract_kernel<true>;
  if ((rc = set_smem(gk, gsm_k)) || (rc = set_smem(ck, csm))) return rc;
  if (tc_mode) {
    const void* tk[4] = {(const void*)mr_contract_tc_kernel<false, false>, (const void*)mr_contract_tc_kernel<false, true>,
                         (const void*)mr_contract_tc_kernel<true, false>, (const void*)mr_contract_tc_kernel<true, true>};
    for (const void* k : tk)
      if ((rc = set_smem(k, sizeof(TCShared)))) return rc;
  }
  const int chunk = std::min(n_elem, kElemChunk);
  float* Kel = nullptr;
  if ((rc = gfe::scratch_alloc((void**)&Kel, sizeof(float) * (size_t)n_elem * kKelF, s, "element matrices"))) return rc;
  float* gpbuf = nullptr;
  if ((rc = gfe::scratch_alloc((void**)&gpbuf, sizeof(float) * (size_t)chunk * kGPItem + 16, s,
                               "Gauss-point tangent blocks"))) {
    gfe::scratch_free(Kel, s);
    return rc;
  }
  unsigned* err = gfe::device_error_word();
  void* prof = gfe::stage_begin(GFE_STAGE_MR_JACOBIAN, s);
  int launches = 0;
  const int sms = gfe::sm_count();
  for (int c0 = 0; c0 < n_elem; c0 += chunk) {
    const int cnt = std::min(chunk, n_elem - c0);
    const int ggrid = (cnt + kGPElems - 1) / kGPElems;
    if (mode == 0)
      mr_gp_kernel<false><<<ggrid, kGPThreads, gsm_k, s>>>(elems + c0, cnt, eq2, elin, nq2, xg, dep, cpar, TK, gpbuf, err);
    else
      mr_gp_kernel<true><<<ggrid, kGPThreads, gsm_k, s>>>(elems + c0, cnt, eq2, elin, nq2, xg, dep, cpar, TK, gpbuf, err);
    launches += 2;
    if (tc_mode) {
      const int tgrid = std::min(cnt, 2 * sms);
      if (mode == 0) {
        if (tc_mode == GFE_TC_TF32X3) launch_contract_tc<false, true>(tgrid, s, elems + c0, cnt, T, gpbuf, Kel, err);
        else launch_contract_tc<false, false>(tgrid, s, elems + c0, cnt, T, gpbuf, Kel, err);
      } else {
        if (tc_mode == GFE_TC_TF32X3) launch_contract_tc<true, true>(tgrid, s, elems + c0, cnt, T, gpbuf, Kel, err);
        else launch_contract_tc<true, false>(tgrid, s, elems + c0, cnt, T, gpbuf, Kel, err);
      }
      continue;
    }
    const int cgrid = std::min((cnt + 1) / 2, 2 * sms);
    if (mode == 0)
      mr_contract_kernel<false><<<cgrid, kCThreads, csm, s>>>(elems + c0, cnt, T, gpbuf, Kel);
    else
      mr_contract_kernel<true><<<cgrid, kCThreads, csm, s>>>(elems + c0, cnt, T, gpbuf, Kel);
  }
  gfe::scratch_free(gpbuf, s);
  if (values && (rc = gather_rows<float>(n_elem, elems, eq2, elin, nq2, nlin, Kel, slots, row_ptr, values, s, err))) {
    gfe::scratch_free(Kel, s);
    return rc;
  }
  if (K_out) {
    const size_t n = (size_t)n_elem * ND * ND;
    widen_element_matrices<<<8 * sms, 256, 0, s>>>(Kel, n, K_out);
    ++launches;
  }
  gfe::stage_end(GFE_STAGE_MR_JACOBIAN, prof, s, launches + (values ? 3 : 0));
  gfe::scratch_free(Kel, s);
  GFE_LAUNCH_CHECK(fn);
  return GFE_OK;
}

int jacobian_entry_point(int mode, int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin,
                         const double* xg, const int32_t* color_elems, const int32_t* color_ptr_host,
                         int32_t n_colors, const double* dep, const double* cpar, const int32_t* slots,
                         const int32_t* row_ptr, double* values, int64_t nnz, double* K_out, int32_t precision,
                         void* stream, const char* fn) {
  int rc = check_mesh(n_elem, eq2, elin, nq2, nlin, xg, fn);
  if (rc) return rc;
  if (!dep || !cpar || (n_elem > 0 && (!color_elems || !color_ptr_host || n_colors <= 0)))
    return gfe::set_error(GFE_ERR_ARG, "%s: invalid arguments", fn);
  if (!K_out && !values) return gfe::set_error(GFE_ERR_ARG, "%s: need CSR values or K_out", fn);
  if (values && (!slots || !row_ptr || nnz < 0))
    return gfe::set_error(GFE_ERR_ARG, "%s: CSR values need the slot map and row_ptr", fn);
  if (color_ptr_host[0] != 0 || color_ptr_host[n_colors] != n_elem)
    return gfe::set_error(GFE_ERR_ARG, "%s: colour offsets must run from 0 to n_elem", fn);
  if (precision != GFE_FP64 && precision != GFE_MIXED && precision != GFE_TC_TF32X3 && precision != GFE_TC_TF32)
    return gfe::set_error(GFE_ERR_ARG, "%s: precision must be GFE_FP64, GFE_MIXED, GFE_TC_TF32X3 or GFE_TC_TF32", fn);
  cudaStream_t s = gfe::as_stream(stream);
  if (precision == GFE_FP64)
    return jacobian_f64(mode, n_elem, eq2, elin, nq2, nlin, xg, color_elems, dep, cpar, slots, row_ptr, values, K_out, s,
                        fn);
  return jacobian_f32(mode, n_elem, eq2, elin, nq2, nlin, xg, color_elems, dep, cpar, slots, row_ptr, values, K_out, s,
                      fn, precision == GFE_MIXED ? 0 : precision);
}

}  // namespace

extern "C" int gfe_mr_jacobian(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin,
                               const double* xg, const int32_t* color_elems, const int32_t* color_ptr_host,
                               int32_t n_colors, const double* dep, const double* cpar, const int32_t* slots,
                               const int32_t* row_ptr, double* values, int64_t nnz, double* K_out, int32_t precision,
                               void* stream) {
  return jacobian_entry_point(0, n_elem, eq2, elin, nq2, nlin, xg, color_elems, color_ptr_host, n_colors, dep, cpar,
                              slots, row_ptr, values, nnz, K_out, precision, stream, "gfe_mr_jacobian");
}

extern "C" int gfe_mr_tangent(int32_t n_elem, const int32_t* eq2, const int32_t* elin, int32_t nq2, int32_t nlin,
                              const double* xg, const int32_t* color_elems, const int32_t* color_ptr_host,
                              int32_t n_colors, const double* dep, const double* cpar, const int32_t* slots,
                              const int32_t* row_ptr, double* values, int64_t nnz, double* K_out, int32_t precision,
                              void* stream) {
  return jacobian_entry_point(1, n_elem, eq2, elin, nq2, nlin, xg, color_elems, color_ptr_host, n_colors, dep, cpar,
                              slots, row_ptr, values, nnz, K_out, precision, stream, "gfe_mr_tangent");
}
