// krylov_resident.cuh -- CG and MINRES iterations in one resident (cooperative) kernel.
//
// On systems whose matrix sits in the L2 (129 MB) an iteration of the launch-per-phase form is mostly
// latency: each of its two or three kernels is launched, ends in a reduction by its last block and
// leaves the SMs idle meanwhile.  Here one launch runs many iterations: one CTA an SM (fewer for small
// systems) and two grid barriers an iteration, at which every CTA leaves its partial sums.  Every CTA adds
// them in one order, so all take the same decisions and the iterates do not depend on scheduling.  What
// bounds an iteration is its chain of dependent steps (measured: a barrier 3,000 cycles, an FP64 add with its
// shuffle 90, an L2 load 700), so the chain is kept short:
//  * a CTA keeps its share of the matrix in shared memory (up to kResSmem) and a thread the vector entries of
//    its rows in registers; only the vector that the products gather goes through the L2;
//  * FP64 scalar work runs in one warp, which hands the workers their factors in the vector type;
//  * CG keeps q = A p by its recurrence q = A z + beta q beside p = z + beta p, so the product takes z,
//    which is final one barrier earlier than beta;
//  * MINRES forms A z without the factor 1 / gamma, which enters afterwards; a warp of its own forms the
//    plane rotation during the product and the first barrier, and the w / x update it belongs to runs
//    with the next Lanczos update.
// (Slots that carry a barrier's number beside the value, read until all are current, save a round trip to the
// L2 but have every CTA poll every slot: slower, 16 instead of 10 us an iteration.)
// Measured, launched form -> resident: CG on the 64^3 Laplace system, FP32 matrix, 42 -> 12.3 us an iteration (the
// sliced-ELL copy 47 MB, of which 32 MB are held on chip), FP64 52 -> 29 us (bound by the FP64 pipe); MINRES on the 8^3
// Mooney-Rivlin tangent, FP32, 24 -> 9.4 us an iteration, on the 13^3 one (93 MB) 38 -> 17.  MINRES chains two FP64 sums
// and two barriers behind 2 us of product.
// A wait is bounded; when it runs out every CTA leaves and the solve returns GFE_ERR_TIMEOUT.
#pragma once

namespace {

// more warps hide the product's loads: at 768 threads an iteration at 64^3 took a fifth longer
constexpr int kCgThreads = 1024;
constexpr int kMinresThreads = 768;  // 80 registers a thread, no spills: the waits invalidate the L1, so that a spill
                                     // costs an L2 round trip an iteration
constexpr int kResPolls = 1 << 21;  // about a second
constexpr int kResMaxGrid = 160;    // CTAs at most
constexpr int kResSmem = 212 << 10; // shared memory for the matrix
constexpr int kCgSmem = 224 << 10;     // of the CG kernel
template <int R>
constexpr int kCgAt = (R * (kCgThreads / 32 - 1) + 1 + 3) / 4 * 4;  // slice bounds of a CTA
constexpr int kCgRows = kCgThreads - 32;
constexpr int kCgWorkers = kCgThreads / 32 - 1;      // worker warps of the CG kernel, then the barrier warp
constexpr int kMinresWorkers = kMinresThreads / 32 - 2;  // of MINRES, then the rotation and the barrier warp

// barrier state of a solve, cleared before each launch: arrivals, and the CTAs' partial sums of the
// iteration's two barriers (the second one's may be two)
struct ResBarrier {
  unsigned count, abort;
  double a[kResMaxGrid], b[2][kResMaxGrid];
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(unsigned* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// The barrier warp (all lanes): publishes v[NV] (lane 0's) in `red`, arrives, waits for every CTA and leaves the
// lane's share of their sums in v.  The CTA's earlier writes are ordered before it by the caller's
// __syncthreads; what other CTAs wrote before theirs may be read after the caller's next __syncthreads.
// False when the wait ran out or another CTA gave up.
template <int NV>
__device__ __forceinline__ bool res_barrier(ResBarrier* bar, double (*red)[kResMaxGrid], unsigned& target,
                                            double (&v)[NV]) {
  const int lane = threadIdx.x & 31, grid = (int)gridDim.x;
  target += (unsigned)grid;
  bool ok = true;
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) __stcg(&red[k][blockIdx.x], v[k]);
    add_release(&bar->count);
    for (int polls = 0; (int)(ld_acquire(&bar->count) - target) < 0; ++polls) {
      if (polls > kResPolls || ((polls & 1023) == 1023 && ld_acquire(&bar->abort) != 0u)) {
        atomicExch(&bar->abort, 1u);
        ok = false;
        break;
      }
    }
  }
  __syncwarp();  // orders the loads below after lane 0's wait (a shuffle alone orders no memory access)
  ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
  // all loads of the partials in flight before the first addition
  double u[NV][kResMaxGrid / 32];
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int i = 0; i < kResMaxGrid / 32; ++i) u[k][i] = lane + 32 * i < grid ? __ldcg(&red[k][lane + 32 * i]) : 0.0;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = u[k][0];
#pragma unroll
    for (int i = 1; i < kResMaxGrid / 32; ++i)
      if (32 * i < grid) v[k] += u[k][i];
  }
  return ok;
}

// CTA barrier that also brings each warp's lanes together again: a warp left diverged by a branch of lane 0
// takes about 600 cycles for each of its shuffles
__device__ __forceinline__ void cta_sync() {
  __syncwarp();
  __syncthreads();
  __syncwarp();
}

template <typename T>
__device__ __forceinline__ T warp_sum_down(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// the lanes' shares of a grid sum added; valid in lane 0.  A small grid takes only the levels it needs.
__device__ __forceinline__ double lanes_sum(double s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < (int)gridDim.x) s += __shfl_down_sync(0xffffffffu, s, o);
  return s;
}
// sum of the worker warps' partials (converted here, once, rather than by every warp); valid in lane 0
template <typename TV>
__device__ __forceinline__ double cta_sum(const TV* part, int workers) {
  const int lane = threadIdx.x & 31;
  double s = lane < workers ? (double)part[lane] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  return s;
}

// ---- CG ---------------------------------------------------------------------------------------------

// At most `iters` iterations from r, z = dinv r, p, q = A p (neither read when `fresh`) and the scalars of *sc
// (beta for the first direction); the state is left for another call.  A warp takes R slices of 32 rows.
template <typename TM, typename TV, typename IT, int R>
__global__ void __launch_bounds__(kCgThreads, 1)
cg_resident(int n, SellMatrix<TM, IT> A, TV* x, TV* r, TV* z, TV* p, TV* q, const TV* __restrict__ dinv,
            const uint8_t* __restrict__ fixed, Scalars* sc, ResBarrier* bar, int iters, bool fresh) {
  extern __shared__ __align__(16) unsigned char res_smem[];
  TV* const s_x = reinterpret_cast<TV*>(res_smem);  // [R][kCgRows] each
  TV* const s_d = s_x + R * kCgRows;
  int* const s_at = reinterpret_cast<int*>(s_d + R * kCgRows);  // first entry of each slice, and the end
  TM* const s_val = reinterpret_cast<TM*>(s_at + kCgAt<R>);
  const int cap = (int)(res_smem + kCgSmem - reinterpret_cast<unsigned char*>(s_val)) / (int)(sizeof(TM) + sizeof(IT));
  IT* s_col = reinterpret_cast<IT*>(s_val + cap);
  __shared__ TV part[2][32];
  __shared__ TV beta_v, alpha_v;
  __shared__ int done, aborted;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool worker = warp < kCgWorkers;
  unsigned target = 0;
  // barrier warp, lane 0
  double beta = 0.0, alpha = 0.0, rz = 0.0, rr = 0.0, tol2 = 0.0, sums[2] = {0.0, 0.0};
  int it = 0, bad = 0;
  if (!worker) {
    tol2 = sc->tol2;
    beta = sc->beta;
    rz = sc->rz;
    if (lane == 0) {
      beta_v = (TV)beta;
      alpha_v = TV(0);
      done = sc->done;
      aborted = 0;
    }
  }
  // this CTA's contiguous, equal share of the slices; as much of it as fits goes to shared memory
  const int slices = (n + kSell - 1) / kSell;
  const int s0 = (int)((long long)slices * blockIdx.x / gridDim.x);
  const int s1 = (int)((long long)slices * (blockIdx.x + 1) / gridDim.x);
  const long long e0 = s0 < s1 ? __ldg(A.sptr + s0) : 0;
  const int held = s0 < s1 ? (int)min((long long)cap, __ldg(A.sptr + s1 - 1) + __ldg(A.slen + s1 - 1) - e0) : 0;
  for (int i = threadIdx.x; i < held; i += kCgThreads) {
    s_val[i] = __ldg(A.val + e0 + i);
    s_col[i] = __ldg(A.col + e0 + i);
  }
  // a thread's rows: slices s0 + u kCgWorkers + warp.  Their bounds, x and 1 / diagonal stay in shared memory, z is
  // formed again from r, so that 64 registers hold the rest: the waits invalidate the L1, and with spilled values an
  // iteration at 64^3 took 16.6 us instead of 12.3.  (Copying the part of z that the CTA's rows read to shared memory
  // first: 15.2 us, for the matrix then has less of it.)
  for (int i = threadIdx.x; i <= s1 - s0; i += kCgThreads)
    s_at[i] = (int)((s0 + i < slices ? __ldg(A.sptr + s0 + i) : __ldg(A.sptr + slices - 1) + __ldg(A.slen + slices - 1)) - e0);
  TV rv[R], pv[R], qv[R], wv[R];
  unsigned off = 0, own = 0;  // bit u: row u is fixed, row u exists
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int sl = s0 + u * kCgWorkers + warp, i = sl * kSell + lane;
    rv[u] = pv[u] = qv[u] = wv[u] = TV(0);
    if (!worker) continue;
    s_x[u * kCgRows + threadIdx.x] = s_d[u * kCgRows + threadIdx.x] = TV(0);
    if (sl < s1 && i < n) {
      own |= 1u << u;
      s_x[u * kCgRows + threadIdx.x] = x[i];
      s_d[u * kCgRows + threadIdx.x] = dinv[i];
      rv[u] = r[i];
      if (!fresh) {
        pv[u] = p[i];
        qv[u] = q[i];
      }
      if (fixed && fixed[i]) off |= 1u << u;
    }
  }
  cta_sync();
  for (int t = 0;; ++t) {
    const bool last = t == iters;
    if (worker) {
      // w = A z (0 on fixed rows), a lane a row
      if (!last) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
          TV acc = TV(0);
          const int sl = u * kCgWorkers + warp, self = (s0 + sl) * kSell + lane;
          const int at = sl < s1 - s0 ? s_at[sl] : 0, len = sl < s1 - s0 ? (s_at[sl + 1] - at) / kSell : 0;
          const bool in_smem = at + len * kSell <= held;  // uniform over the warp
          const TM* va = (in_smem ? s_val + at : A.val + e0 + at) + lane;
          const IT* ca = (in_smem ? s_col + at : A.col + e0 + at) + lane;
          for (int k0 = 0; k0 < len; k0 += kSellUnroll) {
            TM v[kSellUnroll];
            IT cc[kSellUnroll];
#pragma unroll
            for (int k = 0; k < kSellUnroll; ++k) {
              const bool in = k0 + k < len;
              v[k] = in ? va[(k0 + k) * kSell] : TM(0);
              cc[k] = in ? ca[(k0 + k) * kSell] : SellIndex<IT>::pad;
            }
#pragma unroll
            for (int k = 0; k < kSellUnroll; ++k)
              if (cc[k] != SellIndex<IT>::pad) acc += (TV)v[k] * z[SellIndex<IT>::column(cc[k], self)];
          }
          wv[u] = (off >> u) & 1 ? TV(0) : acc;
        }
      }
    } else if (t > 0) {
      // <r, z> and <r, r> of the finished iteration: beta, convergence
      const double rzn = lanes_sum(sums[0]), rrn = lanes_sum(sums[1]);
      rr = rrn;
      ++it;
      beta = rz != 0.0 ? rzn / rz : 0.0;
      rz = rzn;
      if (lane == 0) {
        beta_v = (TV)beta;
        if (!isfinite(rrn)) { bad = 1; done = 1; }
        if (rrn <= tol2) done = 2;
      }
    }
    cta_sync();
    if (done || aborted || last) break;
    if (worker) {
      const TV b = beta_v;
      const bool start = fresh && t == 0;
      TV dot = TV(0);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const TV zv = s_d[u * kCgRows + threadIdx.x] * rv[u];
        pv[u] = start ? zv : zv + b * pv[u];
        qv[u] = start ? wv[u] : wv[u] + b * qv[u];
        if ((own >> u) & 1) dot += pv[u] * qv[u];
      }
      dot = warp_sum_down(dot);
      if (lane == 0) part[0][warp] = dot;
    }
    cta_sync();
    if (!worker) {
      double s[1] = {cta_sum(part[0], kCgWorkers)};
      const bool ok = res_barrier(bar, &bar->a, target, s);
      const double pq = lanes_sum(s[0]);
      alpha = pq != 0.0 ? rz / pq : 0.0;
      if (lane == 0) {
        alpha_v = (TV)alpha;
        if (!(pq > 0.0) || !isfinite(pq)) { bad = 1; done = 1; }
        if (!ok) aborted = 1;
      }
    }
    cta_sync();
    if (done || aborted) break;
    if (worker) {
      const TV a = alpha_v;
      TV sz = TV(0), sr = TV(0);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        s_x[u * kCgRows + threadIdx.x] += a * pv[u];
        rv[u] -= a * qv[u];
        const TV zv = s_d[u * kCgRows + threadIdx.x] * rv[u];
        if ((own >> u) & 1) {
          z[(s0 + u * kCgWorkers + warp) * kSell + lane] = zv;
          sz += rv[u] * zv;
          sr += rv[u] * rv[u];
        }
      }
      sz = warp_sum_down(sz);
      sr = warp_sum_down(sr);
      if (lane == 0) {
        part[0][warp] = sz;
        part[1][warp] = sr;
      }
    }
    cta_sync();
    if (!worker) {
      sums[0] = cta_sum(part[0], kCgWorkers);
      sums[1] = cta_sum(part[1], kCgWorkers);
      if (!res_barrier(bar, bar->b, target, sums) && lane == 0) aborted = 1;
    }
    cta_sync();  // z of every CTA is in place
  }
#pragma unroll
  for (int u = 0; u < R; ++u)
    if ((own >> u) & 1) {
      const int i = (s0 + u * kCgWorkers + warp) * kSell + lane;
      x[i] = s_x[u * kCgRows + threadIdx.x];
      r[i] = rv[u];
      p[i] = pv[u];
      q[i] = qv[u];
    }
  if (blockIdx.x == 0 && !worker && lane == 0) {
    sc->beta = beta;
    sc->alpha = alpha;
    sc->rz = rz;
    if (it > 0) sc->rr = rr;
    sc->it += it;
    if (bad) sc->bad = 1;
    if (aborted) { sc->bad = 2; sc->done = 1; }
    else sc->done = done;
  }
}

// ---- MINRES -----------------------------------------------------------------------------------------

// First group of CTA b: shares of equal cost, a group costing its entries plus c0.  With equal numbers of groups the
// CTAs with the longest rows (a triquadratic node has 89 to 402 entries, by lines of the mesh) held the others up at
// the first barrier: an FP64 Newton solve at 8^3, bound by the FP64 pipe, takes 45.6 instead of 51.0 ms.  An FP32
// group costs its latency more than its entries: with 32 entries' worth as in FP64 an iteration took 10.4 us, with
// 256 it takes the 9.4 of equal numbers.  (Between 3^3 and 13^3 a quarter of either value changes an iteration by -7
// to +6 %, four times by -10 to +16 %.)  `nodes` groups of NC rows, then single rows; e0, total: entries of the nodes'
// rows of one component, and the cost of all groups.
template <int NC>
__device__ int minres_share(const int32_t* __restrict__ rp, int nodes, int n_groups, long long e0, long long c0,
                            long long total, int b, int grid) {
  const long long want = total * b / grid;
  int lo = 0, hi = n_groups;  // the first group with cost(g) >= want
  while (lo < hi) {
    const int g = lo + (hi - lo) / 2;
    const long long e = g <= nodes ? __ldg(rp + g) - 1ll
                                   : e0 + __ldg(rp + g + (NC - 1) * nodes) - __ldg(rp + NC * nodes);
    if (e + c0 * g < want) lo = g + 1;
    else hi = g;
  }
  return lo;
}

// At most `iters` iterations of the preconditioned MINRES from z = Z[j0 & 1] and the scalars of *sc
// (nothing pending); vectors rotate with the iteration number as in the launched form.  NC rows a group:
// the NC components of a node (minres_spmv_nodal), or 1.  A CTA takes a contiguous share of the groups, at
// most kMinresWorkers * 32 rows (the host sees to n_groups / grid + 4 <= kMinresWorkers * 32 / NC), and LPR lanes a
// group in the product.
template <typename TM, typename TV, typename TX, int LPR, int NC>
__global__ void __launch_bounds__(kMinresThreads, 1)
minres_resident(int n, int n_node, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                const TM* __restrict__ val, const uint8_t* __restrict__ fixed, const TV* __restrict__ minv, TX* x,
                TV* V0, TV* V1, TV* Z0, TV* Z1, TV* W0, TV* W1, MinresScalars* sc, ResBarrier* bar, int j0,
                int iters) {
  constexpr int kWorkers = kMinresWorkers;
  extern __shared__ __align__(16) unsigned char res_smem[];
  __shared__ TV q_s[kWorkers * 32];                               // A z on the CTA's rows
  __shared__ TV part[32];
  __shared__ MinresScalars S;                                     // the rotation warp's; S.delta the barrier warp's
  __shared__ TV f_zs, f_a1i, f_a2, f_a3, f_ce, f_g, f_a, f_b;     // the workers' factors
  __shared__ double ig, ig_old, g2_new;                           // 1 / gamma, 1 / gamma_old, gamma^2 just summed
  __shared__ int done, aborted, pending;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool worker = warp < kWorkers, rotation = warp == kWorkers, barrier = warp == kWorkers + 1;
  unsigned target = 0;
  double sums[1] = {0.0};
  if (barrier && lane == 0) {
    S = *sc;
    ig = 1.0 / S.gamma;
    ig_old = 1.0 / S.gamma_old;
    done = S.done;
    aborted = pending = 0;
  }
  // groups [g_begin, g_end) of this CTA: nn nodes, then single rows; their rows are local 0 .. rows - 1,
  // component by component
  const int n_groups = n - (NC - 1) * n_node;
  // c0: as minres_share says, and enough for a share's rows to have a thread each
  __shared__ int g_cut[2];
  if (threadIdx.x < 2) {
    const int nodes = NC > 1 ? n_node : n_groups, grid = (int)gridDim.x;
    const long long e0 = __ldg(rp + nodes) - 1ll, E = e0 + (NC > 1 ? __ldg(rp + n) - __ldg(rp + NC * n_node) : 0);
    const int room = kMinresWorkers * 32 / NC - n_groups / grid - 3;
    const long long c0 = max(sizeof(TV) == 8 ? 32ll : 256ll, (E / grid + 1) / room + 1);
    g_cut[threadIdx.x] = minres_share<NC>(rp, nodes, n_groups, e0, c0, E + c0 * n_groups, blockIdx.x + threadIdx.x, grid);
  }
  __syncthreads();
  const int g_begin = g_cut[0], g_end = g_cut[1];
  const int nn = NC > 1 ? min(max(n_node - g_begin, 0), g_end - g_begin) : 0;
  const int rows = nn * NC + (g_end - g_begin - nn);
  // entries: the nodes' rows are NC contiguous ranges of the CSR, the single rows another one; held in
  // shared memory one after the other as far as they fit
  const int n0 = nn > 0 ? __ldg(rp + g_begin) - 1 : 0, nlen = nn > 0 ? __ldg(rp + g_begin + nn) - 1 - n0 : 0;
  const int single0 = g_begin + nn + (NC - 1) * n_node, singles = g_end - g_begin - nn;  // first single row
  const int m0 = singles > 0 ? __ldg(rp + single0) - 1 : 0;
  const int mlen = singles > 0 ? __ldg(rp + single0 + singles) - 1 - m0 : 0;
  // held entries: the nodes' NC values and columns, then the single rows' values and columns
  const int hn = min(nlen, (int)(kResSmem / (NC * sizeof(TM) + 4)));
  TM* const nv = reinterpret_cast<TM*>(res_smem);
  int32_t* const ncol = reinterpret_cast<int32_t*>(nv + NC * hn);
  const int used = (hn * (int)(NC * sizeof(TM) + 4) + 7) / 8 * 8;
  const int hm = min(mlen, max(0, (kResSmem - used) / (int)(sizeof(TM) + 4)));
  TM* const mv = reinterpret_cast<TM*>(res_smem + used);
  int32_t* const mcol = reinterpret_cast<int32_t*>(mv + hm);
  for (int i = threadIdx.x; i < hn; i += kMinresThreads) ncol[i] = __ldg(ci + n0 + i);
  if (nn > 0)
    for (int c = 0; c < NC; ++c) {
      const TM* v = val + (__ldg(rp + g_begin + (size_t)c * n_node) - 1);
      for (int i = threadIdx.x; i < hn; i += kMinresThreads) nv[c * hn + i] = __ldg(v + i);
    }
  for (int i = threadIdx.x; i < hm; i += kMinresThreads) {
    mcol[i] = __ldg(ci + m0 + i);
    mv[i] = __ldg(val + m0 + i);
  }
  // this thread's row and its vector entries
  const int lr = threadIdx.x;
  const bool own = worker && lr < rows;
  int row = 0;
  TV v_cur = TV(0), v_old = TV(0), z_cur = TV(0), z_old = TV(0), w_new = TV(0), w_old = TV(0), mi = TV(0);
  TX xv = TX(0);
  bool row_fixed = false;
  if (own) {
    row = lr < nn * NC ? g_begin + lr % nn + (lr / nn) * n_node : single0 + lr - nn * NC;
    const bool odd = j0 & 1;
    v_cur = (odd ? V1 : V0)[row];
    v_old = (odd ? V0 : V1)[row];
    z_cur = (odd ? Z1 : Z0)[row];
    z_old = (odd ? Z0 : Z1)[row];
    w_old = (odd ? W1 : W0)[row];
    w_new = (odd ? W0 : W1)[row];
    mi = minv[row];
    xv = x[row];
    row_fixed = fixed && fixed[row];
  }
  constexpr int GPW = 32 / LPR;  // groups a warp
  const int sub = lane % LPR;
  // bounds of the first group of this lane (the later ones, if any, are read again each time)
  auto bounds = [&](int grp, int (&k0)[NC], int& len, bool multi) {
    const int r0 = NC > 1 && !multi ? grp + (NC - 1) * n_node : grp;
    k0[0] = __ldg(rp + r0) - 1;
#pragma unroll
    for (int c = 1; c < NC; ++c) k0[c] = multi ? __ldg(rp + r0 + c * n_node) - 1 : 0;
    len = __ldg(rp + r0 + 1) - 1 - k0[0];
  };
  const int grp1 = g_begin + warp * GPW + lane / LPR;
  int k1[NC], len1 = 0;
#pragma unroll
  for (int c = 0; c < NC; ++c) k1[c] = 0;
  if (worker && grp1 < g_end) bounds(grp1, k1, len1, NC > 1 && grp1 < n_node);
  int j = j0;
  cta_sync();
  for (int t = 0;; ++t, ++j) {
    const bool last = t == iters;
    // whether this iteration's product and first barrier run: read here, where no warp writes `done` (the
    // rotation warp does between the next two CTA barriers)
    const bool go = !last && !done;
    const TV* z = j & 1 ? Z1 : Z0;
    if (worker) {
      if (go)
        for (int gb = g_begin + warp * GPW; gb < g_end; gb += kWorkers * GPW) {  // uniform over a warp
          const int grp = gb + lane / LPR;
          const bool valid = grp < g_end, multi = NC > 1 && grp < n_node;
          int k0[NC], len = 0;
#pragma unroll
          for (int c = 0; c < NC; ++c) k0[c] = k1[c];
          if (gb == g_begin + warp * GPW) len = len1;
          else if (valid) bounds(grp, k0, len, multi);
          TV acc[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) acc[c] = TV(0);
          const int so = multi ? k0[0] - n0 : k0[0] - m0;  // place in shared memory
          if (so + len <= (multi ? hn : hm)) {
            const int32_t* col = (multi ? ncol : mcol) + so;
            const TM* v0 = (multi ? nv : mv) + so;
            for (int t0 = sub; t0 < len; t0 += kNodalBatch * LPR) {
              TV g[kNodalBatch];
#pragma unroll
              for (int u = 0; u < kNodalBatch; ++u) {
                const int k = t0 + u * LPR;
                g[u] = k < len ? z[col[k] - 1] : TV(0);
              }
#pragma unroll
              for (int u = 0; u < kNodalBatch; ++u) {
                const int k = t0 + u * LPR;
                if (k < len) {
                  acc[0] += (TV)v0[k] * g[u];
                  if (NC > 1 && multi) {
#pragma unroll
                    for (int m = 1; m < NC; ++m) acc[m] += (TV)v0[m * hn + k] * g[u];
                  }
                }
              }
            }
          } else {
            // rows that shared memory does not hold are read again every iteration: they should stay in the L2 (an
            // 11^3 tangent, 56 MB in FP32: 11.7 us an iteration; 13.9 with evict-first loads, FP64 36 and 57)
            for (int t0 = sub; t0 < len; t0 += kNodalBatch * LPR) {
              int c[kNodalBatch];
              TM v[NC][kNodalBatch];
#pragma unroll
              for (int u = 0; u < kNodalBatch; ++u) {
                const int k = t0 + u * LPR;
                c[u] = k < len ? __ldg(ci + k0[0] + k) : 0;
#pragma unroll
                for (int m = 0; m < NC; ++m) v[m][u] = k < len && (m == 0 || multi) ? __ldg(val + k0[m] + k) : TM(0);
              }
#pragma unroll
              for (int u = 0; u < kNodalBatch; ++u)
                if (c[u] > 0) {
                  const TV zc = z[c[u] - 1];
#pragma unroll
                  for (int m = 0; m < NC; ++m) acc[m] += (TV)v[m][u] * zc;
                }
            }
          }
#pragma unroll
          for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) acc[c] += __shfl_down_sync(0xffffffffu, acc[c], o, LPR);
          if (valid && sub == 0) {
            const int i = grp - g_begin;
            if (NC > 1 && multi) {
#pragma unroll
              for (int c = 0; c < NC; ++c) q_s[c * nn + i] = acc[c];
            } else {
              q_s[nn * NC + i - nn] = acc[0];
            }
          }
        }
    } else if (barrier && t > 0) {
      const double g2 = lanes_sum(sums[0]);
      if (lane == 0) {
        g2_new = g2;
        ig_old = ig;
        ig = g2 > 0.0 ? rsqrt(g2) : 0.0;
      }
    }
    cta_sync();
    TV qv = TV(0);
    if (worker) {
      if (own && go && !row_fixed) qv = q_s[lr];
      const TV dot = warp_sum_down(z_cur * qv);
      if (lane == 0) part[warp] = dot;
    }
    cta_sync();
    if (barrier) {
      // delta_j, once the rows of every CTA are done; the factors of the Lanczos update
      sums[0] = cta_sum(part, kWorkers);
      bool ok = true;
      if (go) ok = res_barrier(bar, &bar->a, target, sums);
      const double d = lanes_sum(sums[0]) * (ig * ig);
      if (lane == 0) {
        f_g = (TV)ig;
        f_a = (TV)(d * ig);
        f_b = (TV)((t > 0 ? g2_new * ig : S.gamma) * ig_old);
        sums[0] = d;  // stored for the rotation after the next barrier
        if (!ok) aborted = 1;
      }
    } else if (rotation && t > 0) {
      // the rotation of the finished iteration (its delta and gamma in S, the new gamma^2 in g2_new)
      if (lane == 0) {
        const double g2 = g2_new, g = S.gamma, d = S.delta;
        const double a0 = S.c * d - S.c_old * S.s * g;
        const double h2 = fma(a0, a0, g2), ia1 = rsqrt(h2);
        if (!(g2 >= 0.0) || !isfinite(g2) || !(h2 > 0.0) || !isfinite(d)) {
          S.bad = 1;
          done = 1;
        } else {
          const double gn = g2 * ig, cn = a0 * ia1, sn = gn * ia1;
          f_a1i = (TV)ia1;
          f_a2 = (TV)(S.s * d + S.c_old * S.c * g);
          f_a3 = (TV)(S.s_old * g);
          f_ce = (TV)(cn * S.eta);
          f_zs = (TV)ig_old;
          S.eta = -sn * S.eta;
          S.gamma_old = g;
          S.gamma = gn;
          S.c_old = S.c;
          S.c = cn;
          S.s_old = S.s;
          S.s = sn;
          S.it += 1;
          pending = 1;
          if (fabs(S.eta) <= S.tol || gn == 0.0) done = 2;
        }
      }
    }
    cta_sync();
    if (aborted) break;
    const bool stop = done || last;
    if (worker && pending) {
      // w / x update of the finished iteration
      const TV wn = (z_old * f_zs - f_a3 * w_old - f_a2 * w_new) * f_a1i;
      w_old = w_new;
      w_new = wn;
      xv += (TX)(f_ce * wn);
    }
    if (stop) break;
    if (worker) {
      const TV vn = f_g * qv - f_a * v_cur - f_b * v_old;
      v_old = v_cur;
      v_cur = vn;
      z_old = z_cur;
      z_cur = mi * vn;
      if (own) (j & 1 ? Z0 : Z1)[row] = z_cur;
      const TV acc = warp_sum_down(z_cur * vn);
      if (lane == 0) part[warp] = acc;
    }
    cta_sync();
    if (barrier) {
      if (lane == 0) {
        S.delta = sums[0];
        pending = 0;
      }
      sums[0] = cta_sum(part, kWorkers);
      if (!res_barrier(bar, bar->b, target, sums) && lane == 0) aborted = 1;
    }
    cta_sync();  // z_{j+1} of every CTA is in place
  }
  // the state, where iteration j finds it
  if (own) {
    const bool odd = j & 1;
    (odd ? V1 : V0)[row] = v_cur;
    (odd ? V0 : V1)[row] = v_old;
    (odd ? Z0 : Z1)[row] = z_old;
    (odd ? W1 : W0)[row] = w_old;
    (odd ? W0 : W1)[row] = w_new;
    x[row] = xv;
  }
  cta_sync();
  if (blockIdx.x == 0 && barrier && lane == 0) {
    S.pending = 0;
    S.done = done;
    if (aborted) { S.bad = 2; S.done = 1; }
    *sc = S;
  }
}

// Cooperative launch of a resident kernel; false when the device cannot hold its grid at once (the caller
// then runs the launched form).
template <typename... Params, typename... Args>
bool launch_resident(void (*kernel)(Params...), int grid, int threads, int smem, cudaStream_t s, Args... args) {
  if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.dynamicSmemBytes = smem;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess;
}

}  // namespace
