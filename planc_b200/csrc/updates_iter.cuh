// updates_iter.cuh -- the iterative factor updates of the planc NTF solver
// family on the device: AO-ADMM (reference ntf/ntfaoadmm.hpp:23-77) and the
// Nesterov-accelerated proximal gradient with its outer extrapolation
// (ntf/ntfnes.hpp:11-166).
//
// Both updates are row-separable: every row of the I_n x k factor solves its
// own small problem with the shared k x k matrix (G + alpha I, or G + lambda I),
// and the rows only meet in global stopping tests (Frobenius norms for ADMM,
// max / min for Nesterov). A warp owns a row (lane c holds columns c and
// c + 32), the k x k matrix sits in shared memory.
//  * AO-ADMM runs its fixed maximum of 5 iterations as 5 launches; the last
//    CTA of each launch sums the per-CTA partial norms in a fixed order and
//    writes the stop flag that makes the remaining launches return at once.
//  * The Nesterov inner loop has a data-dependent length, so it runs inside
//    one thread-block cluster: each step ends with a cluster barrier, before
//    which every CTA stores its partial max / min into the shared memory of
//    every CTA of the cluster (distributed shared memory); after it each CTA
//    combines the partials from its own shared memory. Max and min are exact,
//    so every CTA takes the same decision. No CTA spins on memory; the
//    barrier is the hardware one. A partial slot is double-buffered by step
//    parity: a CTA can be at most one barrier ahead of another, so it never
//    overwrites a slot another CTA has still to read, and no CTA stores into
//    another after the last barrier, so CTAs may leave in any order.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"

namespace pg {

namespace cg = cooperative_groups;

constexpr int kStMaxIter = -10;  // an iterative update reached its step cap

// Shape of the cluster launches: 16 warps per CTA; 8 CTAs (a portable
// cluster) for the global-memory Nesterov loop, and 16 CTAs where the device
// runs clusters of 16 (8 otherwise) for the register-resident kernels.
constexpr int NES_CTAS = 8;
constexpr int NES_CTAS_MAX = 16;
constexpr int NES_THREADS = 512;

// ---------------------------------------------------------------------------
// AO-ADMM
// ---------------------------------------------------------------------------
constexpr int ADMM_WARPS = 8;        // rows in flight per CTA
constexpr int ADMM_MAX_BLOCKS = 296; // 2 CTAs per SM; partial-norm buffer size

// alpha = trace(G) / k (0.01 if not positive) and L = chol(G + alpha I),
// lower (ntfaoadmm.hpp:29-35); resets the stop flag and the CTA counter.
// One CTA. A non-positive pivot (chol() failure in the reference) sets
// kStSingular.
__global__ void __launch_bounds__(256) k_admm_prep(const double* __restrict__ G, int k,
                                                   double* __restrict__ Lg,
                                                   double* __restrict__ scal, int* __restrict__ flag,
                                                   int* __restrict__ counter, int* __restrict__ status) {
  __shared__ double T[kMaxRank * (kMaxRank + 1)];
  __shared__ double s_alpha;
  __shared__ int s_bad;
  constexpr int LD = kMaxRank + 1;
  const int tid = threadIdx.x;
  if (tid == 0) {
    double tr = 0.0;
    for (int i = 0; i < k; ++i) tr += G[i * k + i];
    double a = tr / k;
    s_alpha = (a > 0) ? a : 0.01;
    s_bad = 0;
  }
  __syncthreads();
  for (int e = tid; e < k * k; e += blockDim.x) {
    const int i = e / k, j = e % k;
    T[i * LD + j] = G[e] + (i == j ? s_alpha : 0.0);
  }
  __syncthreads();
  // left-looking (dot-product) Cholesky, column j after columns < j
  for (int j = 0; j < k; ++j) {
    if (tid == 0) {
      double d = T[j * LD + j];
      for (int p = 0; p < j; ++p) d -= T[j * LD + p] * T[j * LD + p];
      if (!(d > 0.0)) s_bad = 1;
      T[j * LD + j] = d > 0.0 ? sqrt(d) : 1.0;
    }
    __syncthreads();
    const double ljj = T[j * LD + j];
    for (int i = j + 1 + tid; i < k; i += blockDim.x) {
      double v = T[i * LD + j];
      for (int p = 0; p < j; ++p) v -= T[i * LD + p] * T[j * LD + p];
      T[i * LD + j] = v / ljj;
    }
    __syncthreads();
  }
  for (int e = tid; e < k * k; e += blockDim.x) {
    const int i = e / k, j = e % k;
    Lg[e] = j <= i ? T[i * LD + j] : 0.0;
  }
  if (tid == 0) {
    scal[0] = s_alpha;
    *flag = 0;
    *counter = 0;
    if (s_bad) atomicCAS(status, 0, kStSingular);
  }
}

// Selects register slot `p` of a lane's row slice with a compile-time index.
template <int PER>
__device__ __forceinline__ double slot_get(const double (&v)[PER], int p) {
  double r = v[0];
#pragma unroll
  for (int q = 1; q < PER; ++q)
    if (p == q) r = v[q];
  return r;
}

// One ADMM iteration over all rows (ntfaoadmm.hpp:40-72):
//   x   = (G + alpha I)^{-1} (m + alpha (h + u))  [two triangular solves]
//   h'  = max(x - u, 0),  u' = (u + h') - x
// plus the four squared norms of the stopping test. Returns at once when the
// previous launch set the stop flag; the last CTA to finish combines the
// per-CTA partials in CTA order and writes the flag for the next launch.
template <int KP>
__global__ void __launch_bounds__(32 * ADMM_WARPS) k_admm_step(
    double* __restrict__ H, double* __restrict__ U, const double* __restrict__ M,
    const double* __restrict__ Lg, const double* __restrict__ scal, int64_t I, int k, double tol,
    int* __restrict__ flag, double* __restrict__ part, int* __restrict__ counter) {
  if (*flag) return;  // written by the previous launch; uniform over the grid
  constexpr int PER = KP / 32;
  constexpr int LD = KP + 1;  // odd stride: row and column walks are conflict-free
  __shared__ double Ls[KP * LD];
  __shared__ double rinv[KP];
  __shared__ double wred[ADMM_WARPS][4];
  __shared__ int s_last;
  for (int e = threadIdx.x; e < k * k; e += blockDim.x) Ls[(e / k) * LD + e % k] = Lg[e];
  if (threadIdx.x < k) rinv[threadIdx.x] = 1.0 / Lg[threadIdx.x * k + threadIdx.x];
  __syncthreads();
  const double alpha = scal[0];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s_fac = 0.0, s_dual = 0.0, s_r = 0.0, s_s = 0.0;
  for (int64_t row = (int64_t)blockIdx.x * ADMM_WARPS + warp; row < I;
       row += (int64_t)gridDim.x * ADMM_WARPS) {
    double h[PER], u[PER], y[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int c = lane + 32 * p;
      h[p] = c < k ? H[row * k + c] : 0.0;
      u[p] = c < k ? U[row * k + c] : 0.0;
      const double m = c < k ? M[row * k + c] : 0.0;
      y[p] = m + alpha * (h[p] + u[p]);
    }
    // forward substitution with L (column-oriented, the order of dtrsm; the
    // diagonal enters as its reciprocal)
    for (int j = 0; j < k; ++j) {
      const double yj = __shfl_sync(0xffffffffu, slot_get<PER>(y, j >> 5), j & 31) * rinv[j];
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int c = lane + 32 * p;
        if (c == j)
          y[p] = yj;
        else if (c > j && c < k)
          y[p] -= yj * Ls[c * LD + j];
      }
    }
    // back substitution with L^T
    for (int j = k - 1; j >= 0; --j) {
      const double xj = __shfl_sync(0xffffffffu, slot_get<PER>(y, j >> 5), j & 31) * rinv[j];
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int c = lane + 32 * p;
        if (c == j)
          y[p] = xj;
        else if (c < j)
          y[p] -= xj * Ls[j * LD + c];
      }
    }
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int c = lane + 32 * p;
      if (c < k) {
        double hn = y[p] - u[p];
        hn = hn > 0.0 ? hn : 0.0;
        const double un = (u[p] + hn) - y[p];
        s_fac = fma(hn, hn, s_fac);
        s_dual = fma(un, un, s_dual);
        const double d = hn - y[p];
        s_r = fma(d, d, s_r);
        const double e = hn - h[p];
        s_s = fma(e, e, s_s);
        H[row * k + c] = hn;
        U[row * k + c] = un;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s_fac += __shfl_xor_sync(0xffffffffu, s_fac, o);
    s_dual += __shfl_xor_sync(0xffffffffu, s_dual, o);
    s_r += __shfl_xor_sync(0xffffffffu, s_r, o);
    s_s += __shfl_xor_sync(0xffffffffu, s_s, o);
  }
  if (lane == 0) {
    wred[warp][0] = s_fac;
    wred[warp][1] = s_dual;
    wred[warp][2] = s_r;
    wred[warp][3] = s_s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int w = 0; w < ADMM_WARPS; ++w)
      for (int q = 0; q < 4; ++q) t[q] += wred[w][q];
    for (int q = 0; q < 4; ++q) part[blockIdx.x * 4 + q] = t[q];
    __threadfence();
    s_last = atomicAdd(counter, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // the last CTA adds the CTAs' partials, in parallel and in a fixed order
  __shared__ double sh[32 * ADMM_WARPS];
  double t[4];
  for (int q = 0; q < 4; ++q) {
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += part[b * 4 + q];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = blockDim.x >> 1; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    t[q] = sh[0];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double facnorm = sqrt(t[0]), dualnorm = sqrt(t[1]);
    const double r = sqrt(t[2]), s = sqrt(t[3]);
    *flag = (r < tol * facnorm && s < tol * dualnorm) ? 1 : 0;
    *counter = 0;
  }
}

// The whole AO-ADMM update of one mode in one cluster, for modes of at most
// R * 16 rows a CTA (every row's h, u and m in registers): alpha and the
// Cholesky factor (each CTA computes the same one), at most 5 ADMM iterations
// whose stopping norms are summed per warp, per CTA (warp order) and over the
// cluster (CTA order) -- the same sums in every CTA, so every CTA takes the
// same decision -- then the column normalisation of the dual variable with
// column sums formed the same way. Writes the new factor (unnormalised) and
// the dual variable.
//
// Bound by latencies: the factor's k dependent columns, a row's 2 k dependent
// substitution steps an iteration, the exchanges over the cluster. So the
// factor is formed right-looking over the whole CTA (a thread keeps its
// entries in registers; two barriers, a square root and a division a column,
// every entry's subtractions in the order of the left-looking sums), and all
// 5 iterations run before the cluster exchanges their 5 sets of norms: when
// an earlier one meets the test (ntfaoadmm.hpp:63-71) the rows start again
// from global memory and run that many. That is rare: a factor is normalised
// after each update, so the next one has to move it back to its scale and
// takes all 5 iterations (none of 175800 updates of random tensors stopped
// earlier). At 300 / 220 rows of rank 24: 42 / 36 us
// (50 with a factor formed by dot products of one thread a pivot and an
// exchange an iteration).
template <int KP, int R>
__global__ void __launch_bounds__(NES_THREADS, 1)
    k_admm_cluster(double* __restrict__ H, double* __restrict__ U, const double* __restrict__ M,
                   const double* __restrict__ G, int64_t I, int k, double tol,
                   int* __restrict__ status) {
  constexpr int PER = KP / 32;
  constexpr int NW = NES_THREADS / 32;
  constexpr int LD = KP + 1;
  constexpr int ITERS = 5;  // admm_iter, ntfaoadmm.hpp:87
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double Ls[KP * LD];
  __shared__ double wred[ITERS][NW][4];
  // per-CTA partials pushed into every CTA of the cluster (remote shared-
  // memory stores before a cluster barrier), read back locally after it
  __shared__ double slot[NES_CTAS_MAX][ITERS * 4];
  __shared__ double tot[ITERS * 4];
  static_assert((NW + NES_CTAS_MAX) * KP <= KP * LD, "column partials must fit in Ls");
  __shared__ double rinv[KP];
  __shared__ double piv[KP];  // the column being eliminated
  __shared__ double s_alpha;
  const int tid = threadIdx.x;
  // alpha = trace(G) / k (0.01 if not positive), L = chol(G + alpha I)
  // (ntfaoadmm.hpp:29-35)
  if (tid < KP) piv[tid] = tid < k ? G[tid * k + tid] : 0.0;
  __syncthreads();
  if (tid == 0) {
    double tr = 0.0;
    for (int i = 0; i < k; ++i) tr += piv[i];
    const double a = tr / k;
    s_alpha = (a > 0) ? a : 0.01;
  }
  __syncthreads();
  const double alpha = s_alpha;
  {
    constexpr int TPR = NES_THREADS / KP;  // threads of a row
    constexpr int E = KP / TPR;            // entries of a thread: columns q, q + TPR, ...
    const int i = tid / TPR, q = tid % TPR;
    double v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int c = q + e * TPR;
      v[e] = (i < k && c <= i) ? G[i * k + c] + (i == c ? alpha : 0.0) : 0.0;
      if (c == 0) piv[i] = v[e];
    }
    __syncthreads();
    bool bad = false;
    for (int j = 0; j < k; ++j) {
      if (tid < KP) {
        const double d = piv[j];
        if (!(d > 0.0)) bad = true;
        const double ljj = d > 0.0 ? sqrt(d) : 1.0;
        if (tid > j) Ls[tid * LD + j] = piv[tid] / ljj;
        // the substitutions multiply by the reciprocal diagonal (as OpenBLAS's
        // triangular-solve kernels do) instead of dividing on their chain
        if (tid == j) rinv[j] = 1.0 / ljj;
      }
      __syncthreads();
      if (i > j) {
        const double l = Ls[i * LD + j];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const int c = q + e * TPR;
          if (c > j && c <= i) {
            v[e] = fma(-l, Ls[c * LD + j], v[e]);
            if (c == j + 1) piv[i] = v[e];
          }
        }
      }
      __syncthreads();
    }
    if (bad && blockIdx.x == 0 && tid == 0) atomicCAS(status, 0, kStSingular);
  }

  const int lane = tid & 31, warp = tid >> 5;
  const int64_t stride = (int64_t)gridDim.x * NW;
  const int64_t row0 = (int64_t)blockIdx.x * NW + warp;
  double h[R][PER], u[R][PER], m[R][PER];
  bool live[R][PER];
  auto load_rows = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int64_t row = row0 + r * stride;
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int c = lane + 32 * p;
        live[r][p] = row < I && c < k;
        h[r][p] = live[r][p] ? H[row * k + c] : 0.0;
        u[r][p] = live[r][p] ? U[row * k + c] : 0.0;
        m[r][p] = live[r][p] ? M[row * k + c] : 0.0;
      }
    }
  };
  // one ADMM iteration of the held rows (ntfaoadmm.hpp:44-61); s4 takes their
  // squared norms of the stopping test
  auto iterate = [&](double (&s4)[4]) {
    double y[R][PER];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p) y[r][p] = m[r][p] + alpha * (h[r][p] + u[r][p]);
    // forward substitution with L, then back substitution with L^T (the
    // column orders of dtrsm), all held rows interleaved; the next step's
    // entries of L are loaded a step ahead, off the chain
    double d = rinv[0], l[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) l[p] = Ls[(lane + 32 * p) * LD];
    for (int j = 0; j < k; ++j) {
      const double dn = rinv[j + 1 < k ? j + 1 : j];
      double ln[PER];
#pragma unroll
      for (int p = 0; p < PER; ++p) ln[p] = Ls[(lane + 32 * p) * LD + j + 1];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double yj = __shfl_sync(0xffffffffu, slot_get<PER>(y[r], j >> 5), j & 31) * d;
#pragma unroll
        for (int p = 0; p < PER; ++p) {
          const int c = lane + 32 * p;
          const double t = fma(-yj, l[p], y[r][p]);
          y[r][p] = c == j ? yj : (c > j && c < k) ? t : y[r][p];
        }
      }
      d = dn;
#pragma unroll
      for (int p = 0; p < PER; ++p) l[p] = ln[p];
    }
#pragma unroll
    for (int p = 0; p < PER; ++p) l[p] = Ls[(k - 1) * LD + lane + 32 * p];
    for (int j = k - 1; j >= 0; --j) {
      const int jn = j > 0 ? j - 1 : 0;
      const double dn = rinv[jn];
      double ln[PER];
#pragma unroll
      for (int p = 0; p < PER; ++p) ln[p] = Ls[jn * LD + lane + 32 * p];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const double xj = __shfl_sync(0xffffffffu, slot_get<PER>(y[r], j >> 5), j & 31) * d;
#pragma unroll
        for (int p = 0; p < PER; ++p) {
          const int c = lane + 32 * p;
          const double t = fma(-xj, l[p], y[r][p]);
          y[r][p] = c == j ? xj : c < j ? t : y[r][p];
        }
      }
      d = dn;
#pragma unroll
      for (int p = 0; p < PER; ++p) l[p] = ln[p];
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p)
        if (live[r][p]) {
          double hn = y[r][p] - u[r][p];
          hn = hn > 0.0 ? hn : 0.0;
          const double un = (u[r][p] + hn) - y[r][p];
          s4[0] = fma(hn, hn, s4[0]);
          s4[1] = fma(un, un, s4[1]);
          const double dr = hn - y[r][p];
          s4[2] = fma(dr, dr, s4[2]);
          const double ds = hn - h[r][p];
          s4[3] = fma(ds, ds, s4[3]);
          h[r][p] = hn;
          u[r][p] = un;
        }
  };
  load_rows();
#pragma unroll 1
  for (int it = 0; it < ITERS; ++it) {
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
    iterate(s4);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int qd = 0; qd < 4; ++qd) s4[qd] += __shfl_xor_sync(0xffffffffu, s4[qd], o);
    if (lane == 0)
#pragma unroll
      for (int qd = 0; qd < 4; ++qd) wred[it][warp][qd] = s4[qd];
  }
  cluster.sync();  // every CTA runs before remote stores; this CTA's norms are there
  if (tid < ITERS * 4) {
    double t = 0.0;
    for (int w = 0; w < NW; ++w) t += wred[tid >> 2][w][tid & 3];
    for (unsigned b = 0; b < cluster.num_blocks(); ++b)
      *cluster.map_shared_rank(&slot[cluster.block_rank()][tid], b) = t;
  }
  cluster.sync();
  if (tid < ITERS * 4) {
    double t = 0.0;
    for (unsigned b = 0; b < cluster.num_blocks(); ++b) t += slot[b][tid];
    tot[tid] = t;
  }
  __syncthreads();
  int run = ITERS;  // iterations of the update
#pragma unroll
  for (int it = ITERS - 2; it >= 0; --it) {
    const double facnorm = sqrt(tot[it * 4]), dualnorm = sqrt(tot[it * 4 + 1]);
    const double rn = sqrt(tot[it * 4 + 2]), sn = sqrt(tot[it * 4 + 3]);
    if (rn < tol * facnorm && sn < tol * dualnorm) run = it + 1;  // ntfaoadmm.hpp:63-71
  }
  if (run < ITERS) {
    load_rows();
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
    for (int it = 0; it < run; ++it) iterate(s4);
  }
  // dual variable column norms (m_ncp_aux.normalize(mode), ntfaoadmm.hpp:74).
  // No CTA needs its Ls once all are here, so its space holds the per-warp
  // column sums and the per-CTA partials the other CTAs push.
  cluster.sync();
  double(*colw)[KP] = reinterpret_cast<double(*)[KP]>(Ls);
  double(*colpart)[KP] = reinterpret_cast<double(*)[KP]>(Ls + NW * KP);
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    double cs = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (live[r][p]) cs = fma(u[r][p], u[r][p], cs);
    colw[warp][lane + 32 * p] = cs;
  }
  __syncthreads();
  if (tid < k) {
    double t = 0.0;
    for (int w = 0; w < NW; ++w) t += colw[w][tid];
    for (unsigned b = 0; b < cluster.num_blocks(); ++b)
      *cluster.map_shared_rank(&colpart[cluster.block_rank()][tid], b) = t;
  }
  cluster.sync();
  double nrm[PER];
#pragma unroll
  for (int p = 0; p < PER; ++p) {
    const int c = lane + 32 * p;
    double t = 0.0;
    if (c < k)
      for (unsigned b = 0; b < cluster.num_blocks(); ++b) t += colpart[b][c];
    nrm[p] = sqrt(t);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t row = row0 + r * stride;
#pragma unroll
    for (int p = 0; p < PER; ++p)
      if (live[r][p]) {
        const int c = lane + 32 * p;
        H[row * k + c] = h[r][p];
        U[row * k + c] = nrm[p] > 0 ? u[r][p] / nrm[p] : u[r][p];
      }
  }
}

// Column 2-norms of an I x k row-major matrix in two launches (per-CTA
// partial sums of squares, then every CTA sums the partials in CTA order and
// scales its own rows): NCPFactors::normalize(int) (ncpfactors.hpp:346-351)
// without keeping lambda.
constexpr int CN_ROWS = 64;
__global__ void __launch_bounds__(256) k_colsumsq_partial(const double* __restrict__ U, int64_t I,
                                                          int k, double* __restrict__ part) {
  __shared__ double red[256];
  const int tid = threadIdx.x;
  const int lanes = 256 / k;  // threads per column
  const int c = tid % k, l = tid / k;
  const int64_t row0 = (int64_t)blockIdx.x * CN_ROWS;
  double s = 0.0;
  if (l < lanes)
    for (int64_t i = row0 + l; i < I && i < row0 + CN_ROWS; i += lanes) s = fma(U[i * k + c], U[i * k + c], s);
  red[tid] = s;
  __syncthreads();
  if (tid < k) {
    double t = 0.0;
    for (int q = 0; q < lanes; ++q) t += red[q * k + tid];
    part[(int64_t)blockIdx.x * k + tid] = t;
  }
}

__global__ void __launch_bounds__(256) k_colnorm_apply(double* __restrict__ U, int64_t I, int k,
                                                       const double* __restrict__ part, int nblk) {
  __shared__ double nrm[kMaxRank];
  if (threadIdx.x < k) {
    double t = 0.0;
    for (int b = 0; b < nblk; ++b) t += part[(int64_t)b * k + threadIdx.x];
    nrm[threadIdx.x] = sqrt(t);
  }
  __syncthreads();
  const int64_t row0 = (int64_t)blockIdx.x * CN_ROWS;
  const int64_t rows = (I - row0) < CN_ROWS ? (I - row0) : CN_ROWS;
  for (int64_t e = threadIdx.x; e < rows * k; e += blockDim.x) {
    const double n = nrm[e % k];
    if (n > 0) U[row0 * k + e] = U[row0 * k + e] / n;
  }
}

// ---------------------------------------------------------------------------
// Nesterov (NTFNES)
// ---------------------------------------------------------------------------
constexpr int NES_MAX_STEPS = 20000;

// Device state of the Nesterov solver object beyond its factor-sized arrays.
struct NesDev {
  double L, mu, lambda, q, inv;  // of the current mode's update
  double step;                   // acceleration step of this iteration
  double cur_err, acc_err;       // error after the sweep / of the extrapolation
  int acc_exp, acc_fails;        // ntfnes.hpp:186-189 (acc_exp starts at 3)
  int accepted;                  // last acceleration kept
  int err_ctr;                   // index slot for the error kernel
  int steps;                     // inner steps of the last update
};

// ntfnes.hpp:25-37
__device__ __forceinline__ double nes_lambda_of(double L, double mu) {
  const double q = L / mu;
  if (q > 1e6) return 10 * mu;
  if (q > 1e3) return mu;
  return mu / 10;
}

// ntfnes.hpp:39-50: root of x^2 + (alpha^2 - q) x - alpha^2 = 0
__device__ __forceinline__ double nes_alpha_of(double alpha, double q) {
  const double a = 1.0, b = alpha * alpha - q, c = -alpha * alpha;
  const double D = b * b - 4 * a * c;
  return (-b + sqrt(D)) / 2;
}

// Number of eigenvalues below sigma of the symmetric tridiagonal matrix with
// diagonal d and squared off-diagonals e2 (both scaled so that no entry
// exceeds 1): the sign changes of the leading minors of T - sigma I
// (p_i+1 = (d_i - sigma) p_i - e_i^2 p_i-1). No division on the chain; a
// vanishing minor counts as a change. Signs and zeros are read from the words,
// off the FP64 pipe, and both minors are rescaled by a power of two every fourth
// step when they have left [2^-300, 2^300]: a step grows the larger of the two
// by 2^2 at most and shrinks it by 2^-165 at most (2^-59 of a shift next to an
// entry, 2^-106 of a cancellation). More shifts a lane (129 sections a round in
// place of 33) were slower: the chains share one warp's issue.
__device__ __forceinline__ double nes_nonzero(double p2, double p1) {
  return ((__double2hiint(p2) & 0x7fffffff) | __double2loint(p2)) == 0 ? p1 * -0x1p-60 : p2;
}
__device__ __forceinline__ int nes_count_below(const double* d, const double* e2, int k, double sigma) {
  double p0 = 1.0, p1 = nes_nonzero(d[0] - sigma, 1.0);
  int cnt = (unsigned)__double2hiint(p1) >> 31;
  auto step = [&](double di, double ei) {
    const double p2 = nes_nonzero(fma(di - sigma, p1, -(ei * p0)), p1);
    cnt += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
    p0 = p1;
    p1 = p2;
  };
  int i = 1;
  for (; i + 4 <= k; i += 4) {
    double di[4], ei[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      di[u] = d[i + u];
      ei[u] = e2[i + u - 1];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) step(di[u], ei[u]);
    const double m = fmax(fabs(p0), fabs(p1));
    const double f = m > 0x1p300 ? 0x1p-300 : m < 0x1p-300 ? 0x1p300 : 1.0;
    p0 *= f;
    p1 *= f;
  }
  for (; i < k; ++i) step(d[i], e2[i - 1]);
  return cnt;
}

// Extreme eigenvalues of the symmetric G (arma::eig_sym, ntfnes.hpp:111-113),
// as LAPACK's symmetric drivers find them: Householder reduction to
// tridiagonal form (Golub & Van Loan, Matrix Computations, 8.3.1), then
// bisection with Sturm counts (ibid., 8.4.1), 32 shifts a round (one per
// lane; warp 0 narrows the smallest eigenvalue, warp 1 the largest). Bound by
// the k - 2 dependent reflections: eight threads per row, two barriers a
// reflection, the short sums taken by every warp redundantly so that they
// need no barrier: 22 us at k = 16 with the four warps that its rows fill
// (cyclic Jacobi rotations, k/2 disjoint ones a round, took 105 us). One CTA.
// Then lambda, q and 1/(L + lambda) of the update (ntfnes.hpp:114-117). For
// mode 0 it also copies the proximal lambda to the previous one
// (ntfnes.hpp:102-104).
constexpr int NES_PREP_THREADS = 512;
inline int nes_prep_threads(int k) { return k <= 8 ? 64 : (8 * k + 31) / 32 * 32; }
__global__ void __launch_bounds__(NES_PREP_THREADS) k_nes_prep(const double* __restrict__ G, int k,
                                                  NesDev* __restrict__ st, int mode,
                                                  const double* __restrict__ prox_lam,
                                                  double* __restrict__ prev_lam) {
  constexpr int LD = kMaxRank + 1;
  __shared__ double A[kMaxRank * LD];
  __shared__ double pv[kMaxRank];                     // p = tau A v of the reflection
  __shared__ double td[kMaxRank], te[kMaxRank];       // diagonal, off-diagonal
  __shared__ double ext[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (mode == 0 && tid < k) prev_lam[tid] = prox_lam[tid];
  for (int e = tid; e < k * k; e += blockDim.x) A[(e / k) * LD + e % k] = G[e];
  __syncthreads();
  const int row = tid >> 3, part = tid & 7;
  for (int j = 0; j + 2 < k; ++j) {
    // v = x + sign(x_0) ||x|| e_0 for x = A(j+1:, j); every warp forms the norm
    const int c0 = j + 1 + lane, c1 = c0 + 32;
    const double x0 = c0 < k ? A[c0 * LD + j] : 0.0, x1 = c1 < k ? A[c1 * LD + j] : 0.0;
    const double tail = fma(x1, x1, lane == 0 ? 0.0 : x0 * x0);
    double s2 = tail;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    const double head = A[(j + 1) * LD + j];
    if (s2 == 0.0) {  // the column is already reduced (the same in every thread)
      if (tid == 0) te[j] = head;
      continue;
    }
    const double nrm = sqrt(fma(head, head, s2));
    const double e = head > 0.0 ? -nrm : nrm;
    const double v_head = head - e;
    const double tau = 2.0 / fma(v_head, v_head, s2);
    auto v_at = [&](int c) { return c == j + 1 ? v_head : A[c * LD + j]; };
    const bool mine = row > j && row < k;
    double acc = 0.0;
    if (mine)
      for (int c = j + 1 + part; c < k; c += 8) acc = fma(A[row * LD + c], v_at(c), acc);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (mine && part == 0) pv[row] = tau * acc;
    if (tid == 0) te[j] = e;
    __syncthreads();
    // K = tau / 2 v^T p, w = p - K v, A -= v w^T + w v^T
    const double vl0 = c0 < k ? (lane == 0 ? v_head : x0) : 0.0, vl1 = x1;
    double vp = fma(vl1, c1 < k ? pv[c1] : 0.0, c0 < k ? vl0 * pv[c0] : 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vp += __shfl_xor_sync(0xffffffffu, vp, o);
    const double K = 0.5 * tau * vp;
    if (mine) {
      const double vr = v_at(row), wr = fma(-K, vr, pv[row]);
      for (int c = j + 1 + part; c < k; c += 8) {
        const double vc = v_at(c), wc = fma(-K, vc, pv[c]);
        A[row * LD + c] -= fma(vr, wc, wr * vc);
      }
    }
    __syncthreads();
  }
  if (tid < k) td[tid] = A[tid * LD + tid];
  if (tid == 0 && k >= 2) te[k - 2] = A[(k - 1) * LD + k - 2];
  __syncthreads();
  if (warp < 2) {
    // a power of two above the Gershgorin bound scales the matrix into [-1, 1]
    double bound = 0.0;
    for (int i = lane; i < k; i += 32)
      bound = fmax(bound, fabs(td[i]) + (i + 1 < k ? fabs(te[i]) : 0.0) + (i > 0 ? fabs(te[i - 1]) : 0.0));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bound = fmax(bound, __shfl_xor_sync(0xffffffffu, bound, o));
    int ex = 0;
    frexp(bound, &ex);
    const double scale = ldexp(1.0, -ex);
    double* d = A + warp * 2 * kMaxRank;  // the reduced matrix is no longer needed
    double* e2 = d + kMaxRank;
    for (int i = lane; i < k; i += 32) {
      const double e = i + 1 < k ? te[i] * scale : 0.0;
      d[i] = td[i] * scale;
      e2[i] = e * e;
    }
    __syncwarp();
    const int want = warp == 0 ? 1 : k;  // smallest: count >= 1; largest: count >= k
    double lo = -1.0, hi = 1.0;
    // 2^-59 of the norm, or two units in the last place: rounds end there
    for (int it = 0; it < 24 && hi - lo > fmax(0x1p-59, 0x1p-52 * fmax(fabs(lo), fabs(hi))); ++it) {
      const double h = (hi - lo) * (1.0 / 33.0);
      const double sg = fma(h, (double)(lane + 1), lo);
      const unsigned b = __ballot_sync(0xffffffffu, nes_count_below(d, e2, k, sg) >= want);
      const int f = b ? __ffs(b) - 1 : 32;  // first shift with enough eigenvalues below it
      const double nh = f < 32 ? fma(h, (double)(f + 1), lo) : hi;
      lo = f > 0 ? fma(h, (double)f, lo) : lo;
      hi = nh;
    }
    // an interval that holds zero at the rounding level of the norm is zero
    const double mid = (lo <= 0.0 && hi >= 0.0) ? 0.0 : 0.5 * (lo + hi);
    if (lane == 0) ext[warp] = ldexp(mid, ex);
  }
  __syncthreads();
  if (tid == 0) {
    const double lo = ext[0], hi = ext[1];
    const double lam = nes_lambda_of(hi, lo);
    st->L = hi;
    st->mu = lo;
    st->lambda = lam;
    st->q = (lo + lam) / (hi + lam);
    st->inv = 1 / (hi + lam);
  }
}

// NTFNES::update inner loop (ntfnes.hpp:100-151) for all rows of one mode,
// in one cluster of NES_CTAS CTAs:
//   prev = H0 = prox;  Ht = acc = H0;  modM = (-lambda) H0 - M
//   loop: grad = modM + (G + lambda I) acc
//         stop if max|grad .* acc| <= 1e-2 and min(grad) >= -1e-2
//         Ht' = max(acc - grad / (L + lambda), 0)
//         alpha, beta (ntfnes.hpp:143-145); acc = Ht' + beta (Ht' - Ht)
// Ht is the mode's factor buffer (the update's output, unnormalised); acc,
// grad and modM are I x k scratch arrays. A step cap (the reference loops
// without one) sets kStMaxIter.
template <int KP>
__global__ void __cluster_dims__(NES_CTAS, 1, 1) __launch_bounds__(NES_THREADS, 1)
    k_nes_inner(double* __restrict__ Ht, const double* __restrict__ prox, double* __restrict__ prev,
                const double* __restrict__ M, const double* __restrict__ G, NesDev* __restrict__ st,
                double* __restrict__ acc, double* __restrict__ grad, double* __restrict__ modM,
                int64_t I, int k, int max_steps, int* __restrict__ status) {
  constexpr int PER = KP / 32;
  constexpr int NW = NES_THREADS / 32;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double Gs[KP * KP];
  __shared__ double wmax[NW], wmin[NW];
  __shared__ double slot[2][NES_CTAS_MAX][2];  // pushed by every CTA, read locally
  const double lam = st->lambda, q = st->q, inv = st->inv;
  for (int e = threadIdx.x; e < k * k; e += NES_THREADS)
    Gs[e] = G[e] + ((e / k) == (e % k) ? lam : 0.0);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t stride = (int64_t)gridDim.x * NW;
  const int64_t row0 = (int64_t)blockIdx.x * NW + warp;
  double vmax = 0.0, vmin = INFINITY;

  // grad = modM + Gs acc for one row (acc in registers), with the row's
  // contribution to the stopping test
  auto row_grad = [&](int64_t row, const double (&a)[PER], const double (&mm)[PER]) {
    double g[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) g[p] = 0.0;
    for (int j = 0; j < k; ++j) {
      const double aj = __shfl_sync(0xffffffffu, slot_get<PER>(a, j >> 5), j & 31);
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int c = lane + 32 * p;
        if (c < k) g[p] = fma(aj, Gs[j * k + c], g[p]);
      }
    }
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int c = lane + 32 * p;
      if (c < k) {
        const double gr = mm[p] + g[p];
        grad[row * k + c] = gr;
        vmax = fmax(vmax, fabs(gr * a[p]));
        vmin = fmin(vmin, gr);
      }
    }
  };

  for (int64_t row = row0; row < I; row += stride) {
    double a[PER], mm[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int c = lane + 32 * p;
      const double h0 = c < k ? prox[row * k + c] : 0.0;
      a[p] = h0;
      mm[p] = c < k ? (-1 * lam) * h0 - M[row * k + c] : 0.0;
      if (c < k) {
        prev[row * k + c] = h0;
        Ht[row * k + c] = h0;
        acc[row * k + c] = h0;
        modM[row * k + c] = mm[p];
      }
    }
    row_grad(row, a, mm);
  }

  double alpha = 1.0, beta = 1.0;
  int t = 0;
  for (;;) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
      vmin = fmin(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
    }
    if (lane == 0) {
      wmax[warp] = vmax;
      wmin[warp] = vmin;
    }
    __syncthreads();
    if (warp == 0) {  // CTA max / min over the warps, pushed to every CTA
      double m = lane < NW ? wmax[lane] : 0.0, n = lane < NW ? wmin[lane] : INFINITY;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        n = fmin(n, __shfl_xor_sync(0xffffffffu, n, o));
      }
      if (lane < (int)cluster.num_blocks()) {
        double* dst = cluster.map_shared_rank(&slot[t & 1][cluster.block_rank()][0], lane);
        dst[0] = m;
        dst[1] = n;
      }
    }
    cluster.sync();
    double gmax = 0.0, gmin = INFINITY;
    for (unsigned r = 0; r < cluster.num_blocks(); ++r) {
      gmax = fmax(gmax, slot[t & 1][r][0]);
      gmin = fmin(gmin, slot[t & 1][r][1]);
    }
    if (gmax <= 1e-2 && gmin >= -1e-2) break;  // stop_iter, ntfnes.hpp:52-62
    if (t >= max_steps) {
      if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(status, 0, kStMaxIter);
      break;
    }
    ++t;
    const double alpha_prev = alpha;
    alpha = nes_alpha_of(alpha_prev, q);
    beta = (alpha_prev * (1 - alpha_prev)) / (alpha + alpha_prev * alpha_prev);
    vmax = 0.0;
    vmin = INFINITY;
    for (int64_t row = row0; row < I; row += stride) {
      double a[PER], mm[PER];
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const int c = lane + 32 * p;
        a[p] = 0.0;
        mm[p] = 0.0;
        if (c < k) {
          const double hprev = Ht[row * k + c];
          const double v = acc[row * k + c] - (inv * grad[row * k + c]);
          const double hn = v > 0.0 ? v : 0.0;
          a[p] = hn + beta * (hn - hprev);
          mm[p] = modM[row * k + c];
          Ht[row * k + c] = hn;
          acc[row * k + c] = a[p];
        }
      }
      row_grad(row, a, mm);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) st->steps = t;
}

// The same loop with every row's state in registers, for modes whose rows fit
// the cluster. A warp holds R groups of rows, 32 / KP rows a group at KP = 16
// and one above, lane c of a row holding column c (and c + 32 at KP = 64).
//
// A step is bound by latencies (a row's k dependent fused multiply-adds, the
// exchange of the stopping test over the cluster), not by a unit, so:
//  * the test is a yes or no (any entry with |grad .* acc| > 1e-2 or grad <
//    -1e-2; NaN counts as passed, as in a max / min), one bit a step, and S
//    steps run before the cluster exchanges their bits: the steps past the
//    one that ends the loop are speculative, and the result is recomputed
//    from the state kept (in shared memory) at the start of its S steps;
//  * the exchange of one group of S steps travels while the next S steps run;
//  * a row's acc reaches its lanes as broadcast 16-byte shared-memory loads
//    (two shuffles per entry would bound the loop), a lane's column of
//    G + lambda I stays in registers where it fits (GREG);
//  * the step lengths beta, a chain of a square root and a division a step,
//    come from one extra warp, S steps ahead.
// Values and step counts are those of the one-step loop, which took 205 us a
// call at 200 x 150 x 120, k = 16 (FP64), against 41 us.
template <int KP, int R>
struct NesReg {
  static constexpr int LPR = KP < 32 ? KP : 32;   // lanes of a row
  static constexpr int RW = 32 / LPR;             // rows of a group
  static constexpr int PER = KP / LPR;            // columns of a lane
  static constexpr int S = R <= 2 ? 4 : 2;        // steps per exchange
  static constexpr bool GREG = KP == 16 || (KP == 32 && R <= 2);
  // warps that hold rows: 15 beside the step-length warp leave 128 registers
  // a thread (room for the column of G + lambda I), 16 leave 96
  static constexpr int NW = R <= 2 ? NES_THREADS / 32 - 1 : NES_THREADS / 32;
  static constexpr int THREADS = (NW + 1) * 32;
  static constexpr int64_t ROWS = (int64_t)NW * RW * R;         // rows of a CTA
  static constexpr size_t ACC = (size_t)NW * R * RW * KP;       // row vectors
  static constexpr size_t KEEP = (size_t)4 * R * PER * NW * 32; // two kept states
  static constexpr size_t SMEM = (ACC + KEEP + (GREG ? 0 : (size_t)KP * KP)) * sizeof(double);
};

template <int KP, int R>
__global__ void __launch_bounds__(NesReg<KP, R>::THREADS, 1)
    k_nes_inner_reg(double* __restrict__ Ht_out, const double* __restrict__ prox,
                    double* __restrict__ prev, const double* __restrict__ M,
                    const double* __restrict__ G, NesDev* __restrict__ st, int64_t I, int k,
                    int max_steps, int* __restrict__ status) {
  using C = NesReg<KP, R>;
  constexpr int PER = C::PER, NW = C::NW, S = C::S;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) double nes_sm[];
  double* arow = nes_sm;                 // [warp][group][row of the group][KP]
  double* keep = arow + C::ACC;          // [parity][ht, acc][group][PER][thread]
  double* Gs = keep + C::KEEP;           // !GREG: G + lambda I, k x k at stride KP
  __shared__ double betas[4][S];
  __shared__ unsigned wmask[2][NW];
  __shared__ unsigned slot[2][NES_CTAS_MAX];  // pushed by every CTA, read locally
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ncta = (int)cluster.num_blocks(), me = (int)cluster.block_rank();
  const double lam = st->lambda, q = st->q, inv = st->inv;
  const bool holder = warp < NW;         // the last warp forms the step lengths
  const int c0 = lane % C::LPR, half = lane / C::LPR;
  auto g_at = [&](int j, int c) {
    return (j < k && c < k) ? G[j * k + c] + (j == c ? lam : 0.0) : 0.0;
  };
  if constexpr (!C::GREG) {
    for (int e = tid; e < KP * KP; e += C::THREADS) Gs[e] = g_at(e / KP, e % KP);
  }
  double greg[C::GREG ? KP : 1];
  if constexpr (C::GREG) {
#pragma unroll
    for (int j = 0; j < KP; ++j) greg[j] = g_at(j, c0);
  }
  double ht[R][PER], acc[R][PER], gr[R][PER], mm[R][PER];
  bool live[R][PER];
  // rows go round the CTAs, so that every CTA holds as many
  auto row_of = [&](int r) {
    return ((int64_t)(r * NW + warp) * ncta + me) * C::RW + half;
  };
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int64_t row = row_of(r);
      const int c = c0 + 32 * p;
      live[r][p] = holder && row < I && c < k;
      const double h0 = live[r][p] ? prox[row * k + c] : 0.0;
      ht[r][p] = h0;
      acc[r][p] = h0;
      mm[r][p] = live[r][p] ? (-1 * lam) * h0 - M[row * k + c] : 0.0;
      gr[r][p] = 0.0;
      if (live[r][p]) prev[row * k + c] = h0;
    }
  const bool working = __any_sync(0xffffffffu, live[0][0]);  // the warp's first group has rows
  double* my_rows = arow + (size_t)(holder ? warp : 0) * R * C::RW * KP;
  // gr = mm + (G + lambda I) acc for every held row (sums over j in order)
  auto all_grads = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p) my_rows[(r * C::RW + half) * KP + c0 + 32 * p] = acc[r][p];
    __syncwarp();
    double g[R][PER];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p) g[r][p] = 0.0;
#pragma unroll
    for (int j = 0; j < KP; j += 4) {
      if (j < k) {
        double gv[4][PER];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int p = 0; p < PER; ++p) {
            if constexpr (C::GREG)
              gv[u][p] = greg[j + u];
            else
              gv[u][p] = Gs[(j + u) * KP + c0 + 32 * p];
          }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const double2* a = reinterpret_cast<const double2*>(my_rows + (r * C::RW + half) * KP + j);
          const double2 a0 = a[0], a1 = a[1];
#pragma unroll
          for (int p = 0; p < PER; ++p) {
            g[r][p] = fma(a0.x, gv[0][p], g[r][p]);
            g[r][p] = fma(a0.y, gv[1][p], g[r][p]);
            g[r][p] = fma(a1.x, gv[2][p], g[r][p]);
            g[r][p] = fma(a1.y, gv[3][p], g[r][p]);
          }
        }
      }
    }
    __syncwarp();  // the rows are read before the next step replaces them
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p) gr[r][p] = mm[r][p] + g[r][p];
  };
  auto step = [&](double beta) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p)
        if (live[r][p]) {
          const double hprev = ht[r][p];
          const double v = acc[r][p] - (inv * gr[r][p]);
          const double hn = v > 0.0 ? v : 0.0;
          acc[r][p] = hn + beta * (hn - hprev);
          ht[r][p] = hn;
        }
    all_grads();
  };
  auto kept = [&](int par, int what, int r, int p) -> double& {
    return keep[(((size_t)par * 2 + what) * R * PER + r * PER + p) * (NW * 32) + tid];
  };
  double alpha = 1.0;
  auto next_betas = [&](int b) {  // ntfnes.hpp:143-145, the last warp
#pragma unroll
    for (int s = 0; s < S; ++s) {
      const double an = nes_alpha_of(alpha, q);
      const double beta = (alpha * (1 - alpha)) / (an + alpha * alpha);
      if (lane == 0) betas[b][s] = beta;
      alpha = an;
    }
  };
  if constexpr (!C::GREG) __syncthreads();
  if (working) all_grads();
  if (!holder) next_betas(0);
  cluster.sync();  // every CTA runs before remote stores; the first betas are there
  int stop_at = 0;   // the step of group `stop_grp` whose state is the result
  int stop_grp = 0;
  for (int grp = 0;; ++grp) {
    if (holder) {
      unsigned bits = 0;
      if (working) {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int p = 0; p < PER; ++p) {
            kept(grp & 1, 0, r, p) = ht[r][p];
            kept(grp & 1, 1, r, p) = acc[r][p];
          }
#pragma unroll 1
        for (int s = 0; s < S; ++s) {
          bool open = false;  // this state does not pass the stopping test
#pragma unroll
          for (int r = 0; r < R; ++r)
#pragma unroll
            for (int p = 0; p < PER; ++p)
              open |= live[r][p] && (fabs(gr[r][p] * acc[r][p]) > 1e-2 || gr[r][p] < -1e-2);
          bits |= open ? 1u << s : 0u;
          step(betas[grp & 3][s]);
        }
        bits = __reduce_or_sync(0xffffffffu, bits);
      }
      if (lane == 0) wmask[grp & 1][warp] = bits;
    } else {
      next_betas((grp + 1) & 3);
    }
    if (grp > 0) {  // the previous group's exchange is complete
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      unsigned open = 0;
      for (int b = 0; b < ncta; ++b) open |= slot[(grp - 1) & 1][b];
      const int first = __ffs(~open) - 1;  // first state that passes (bits >= S are clear)
      const int t0 = (grp - 1) * S;
      if (first < S && first <= max_steps - t0) {  // stop_iter, ntfnes.hpp:52-62
        stop_at = first;
        stop_grp = grp - 1;
        break;
      }
      if (max_steps - t0 < S) {
        stop_at = max_steps - t0;
        stop_grp = grp - 1;
        if (me == 0 && tid == 0) atomicCAS(status, 0, kStMaxIter);
        break;
      }
    }
    __syncthreads();
    if (tid < ncta) {
      unsigned m = 0;
      for (int w = 0; w < NW; ++w) m |= wmask[grp & 1][w];
      *cluster.map_shared_rank(&slot[grp & 1][me], tid) = m;
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  }
  if (!holder) return;
  if (working) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        ht[r][p] = kept(stop_grp & 1, 0, r, p);
        acc[r][p] = kept(stop_grp & 1, 1, r, p);
      }
    if (stop_at > 0) {
      all_grads();
      for (int s = 0; s < stop_at; ++s) step(betas[stop_grp & 3][s]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t row = row_of(r);
#pragma unroll
    for (int p = 0; p < PER; ++p)
      if (live[r][p]) Ht_out[row * k + c0 + 32 * p] = ht[r][p];
  }
  if (me == 0 && tid == 0) st->steps = stop_grp * S + stop_at;
}

// After the mode's normalisation: prox = the normalised factor, and for the
// last mode the proximal lambda = the factor's lambda (normalize_rows of
// m_prox_t, ntfnes.hpp:148-149).
__global__ void __launch_bounds__(256) k_nes_post(const double* __restrict__ F,
                                                  double* __restrict__ prox, int64_t n,
                                                  const double* __restrict__ lambda,
                                                  double* __restrict__ prox_lam, int k) {
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < n; e += (int64_t)gridDim.x * 256)
    prox[e] = F[e];
  if (prox_lam && blockIdx.x == 0 && threadIdx.x < k) prox_lam[threadIdx.x] = lambda[threadIdx.x];
}

// Start of NTFNES::accelerate (ntfnes.hpp:64-75) for the iteration whose
// error was just written: acc_step = (iter + 1)^(1 / acc_exp); keeps the
// current error, lambda and Grams (the state a failed extrapolation returns
// to) and resets the error slot index of the extrapolation's error.
__global__ void __launch_bounds__(256) k_nes_acc_begin(const int* __restrict__ counter,
                                                       const double* __restrict__ errs,
                                                       NesDev* __restrict__ st,
                                                       const double* __restrict__ lambda,
                                                       double* __restrict__ lam_bak,
                                                       const double* __restrict__ Gall,
                                                       double* __restrict__ gall_bak, int nG, int k) {
  if (threadIdx.x == 0) {
    const int iter = *counter - 1;
    st->cur_err = errs[iter];
    st->step = pow((double)(iter + 1), 1.0 / st->acc_exp);
    st->err_ctr = 0;
  }
  if (threadIdx.x < k) lam_bak[threadIdx.x] = lambda[threadIdx.x];
  for (int e = threadIdx.x; e < nG; e += 256) gall_bak[e] = Gall[e];
}

// Extrapolated factor of one mode (ntfnes.hpp:76-88), written over the
// factor: a = cur + step (cur - prv), cur = diag(sc) F, prv = diag(sp) prev,
// with sc / sp the current / previous lambda for the last mode (the only
// unnormalised one) and the identity otherwise.
__global__ void __launch_bounds__(256) k_nes_extrap(double* __restrict__ F,
                                                    const double* __restrict__ prev, int64_t n, int k,
                                                    const double* __restrict__ sc,
                                                    const double* __restrict__ sp,
                                                    const NesDev* __restrict__ st) {
  const double step = st->step;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < n; e += (int64_t)gridDim.x * 256) {
    const int r = (int)(e % k);
    const double cur = sc ? sc[r] * F[e] : F[e];
    const double prv = sp ? sp[r] * prev[e] : prev[e];
    double a = cur - prv;
    a *= step;
    a += cur;
    F[e] = a;
  }
}

// Acceptance test of the extrapolation (ntfnes.hpp:89-98). Rejected: the
// Grams and lambda of the proximal iterate come back (its factors by
// k_nes_commit), the failure count rises and every fail_limit + 1 failures
// the step exponent grows. Accepted: the proximal lambda becomes the norms
// of the (normalised) extrapolated last factor, sqrt(diag G_{N-1}).
__global__ void __launch_bounds__(256) k_nes_decide(NesDev* __restrict__ st,
                                                    double* __restrict__ lambda,
                                                    double* __restrict__ prox_lam,
                                                    double* __restrict__ Gall,
                                                    const double* __restrict__ gall_bak, int nG,
                                                    const double* __restrict__ Glast, int k) {
  __shared__ int s_acc;
  if (threadIdx.x == 0) s_acc = st->acc_err < st->cur_err;
  __syncthreads();
  const int accepted = s_acc;
  if (accepted) {
    if (threadIdx.x < k) prox_lam[threadIdx.x] = sqrt(Glast[threadIdx.x * k + threadIdx.x]);
  } else {
    if (threadIdx.x < k) lambda[threadIdx.x] = prox_lam[threadIdx.x];
    for (int e = threadIdx.x; e < nG; e += 256) Gall[e] = gall_bak[e];
  }
  if (threadIdx.x == 0) {
    st->accepted = accepted;
    if (!accepted) {
      st->acc_fails++;
      if (st->acc_fails > 5) {  // fail_limit, ntfnes.hpp:190
        st->acc_fails = 0;
        st->acc_exp++;
      }
    }
  }
}

// Factor side of the decision for one mode: accepted -> prox = F (the
// extrapolated, normalised factor); rejected -> F = prox.
__global__ void __launch_bounds__(256) k_nes_commit(double* __restrict__ F, double* __restrict__ prox,
                                                    int64_t n, const NesDev* __restrict__ st) {
  const int accepted = st->accepted;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < n; e += (int64_t)gridDim.x * 256) {
    if (accepted)
      prox[e] = F[e];
    else
      F[e] = prox[e];
  }
}

}  // namespace pg
