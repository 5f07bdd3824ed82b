// mode_cluster.cuh -- the end of one factor's step of the outer iteration in
// one cluster launch: [HALS or MU row update, rank <= 16] -> normalisation ->
// Gram -> next leave-one-out product -> [relative error].
//
// Reference: NTFHALS / NTFMU::update (ntf/ntfhals.hpp:13-29, ntf/ntfmu.hpp:
// 11-16), NCPFactors::normalize(int) (common/ncpfactors.hpp:346-351), the Gram
// of the normalised factor and the leave-one-out product
// (common/ncpfactors.hpp:139-148), AUNTF::computeObjectiveError
// (ntf/auntf.hpp:200-246).
//
// What bounds it: a factor is small (I x k doubles), so nothing but the chain
// of dependent steps counts -- launches, trips to L2, barriers, a row's k
// dependent column steps. So the rows stay in shared memory from the update to
// the normalised store, and everything between is one launch.
//
// Layout: a cluster of up to 16 CTAs splits the rows evenly, 64 (16 above rank
// 32) or more a CTA. U^T U of a CTA's rows is summed row by row in increasing
// order on the FP64 tensor cores, an 8 x 8 block of the upper triangle a warp
// (the transposed outputs have the same products in the same order), and over the cluster in rank
// order: the sums, hence the bits, depend on I and k alone, not on the launch
// (alone, or a member of a grouped launch) nor on how the threads share it.
// The update gives a row to 4 lanes, each holding 4 columns in pairs, so that a
// warp carries 8 rows through the recurrence at once; G is read as 16-byte
// loads and only the step's change travels by shuffle; H G starts as tensor-core
// products in the lanes' own layout. Its sums run in the
// order of the one-row-per-warp kernels (the same bits). Above rank 16 the
// loads of G by 16 SMs would cost more than the launch they save (at 1024 rows,
// rank 32: 4.4 us for k_hals_warp over the whole GPU), so the update stays a
// launch of its own there.
// Loads are what a CTA waits for first: the rows, G and M are copied to shared
// memory asynchronously, all in flight together, and the other modes' Grams are
// prefetched meanwhile. Measured a mode: 64^3 rank 8, HALS and every third error
// included, 5.4 us (6.7 with the copies one after another, a division by k for
// every element and the sums by fused multiply-adds, 6.0 without those sums on
// the tensor cores; 2.2 + 8.8 as two launches, and 4.7 a sweep for the error's
// own); without the update, 512 rows of rank 32 8.0 (10.1, 8.8; 11.0 and 9.4),
// 192 rows of rank 64 12.8 (14.7, 13.8).
#pragma once
#include "common.cuh"
#include "updates_iter.cuh"

namespace pg {

enum ModeUpdate { MODE_NONE = 0, MODE_HALS = 1, MODE_MU = 2 };

constexpr int MODE_THREADS = 256;
constexpr int64_t MODE_MAX_ROWS = 4096;
constexpr int MODE_MAX_CL = 16;

struct ModeArgs {
  double* F;             // I x k: the factor, replaced by the normalised update
  const double* M;       // MTTKRP of the mode, I x k (update and error)
  int64_t I;
  int k;
  double eps;            // MU
  double* lambda;
  double* Gall;          // N x k x k Grams
  int N, n, next;        // updated mode; mode whose leave-one-out product is formed (-1: none)
  double* Gloo;          // in: leave-one-out product of mode n; out: of mode next
  int CLm;               // CTAs that hold rows (<= the cluster's size)
  const double* normX2;  // relative error after the update (errs null: none)
  double* errs;
  int* counter;
};

template <int KP>
struct ModeShape {
  static constexpr int LPR = 4;                     // lanes of a row in the update
  static constexpr int CP = KP / LPR;               // columns of a lane
  static constexpr int RPW = 32 / LPR;              // rows of a warp
  static constexpr int CHUNK = RPW * (MODE_THREADS / 32);
  static constexpr int LDH = KP + 2;                // row stride: conflict-free 16-byte rows
  static constexpr int LDG = KP + 4;                // row stride of G: conflict-free fragments
  static constexpr int KB = KP / 8;                 // 8 x 8 blocks of U^T U per edge
  static constexpr int NT = KB * (KB + 1) / 2;      // blocks of its upper triangle
  static constexpr int TPW = (NT + MODE_THREADS / 32 - 1) / (MODE_THREADS / 32);  // a warp's blocks
};

// CTAs of a factor's cluster: one per 64 rows (16 above rank 32, where a
// row's outer product is four times the work)
__host__ __device__ constexpr int mode_ctas(int64_t I, int k, int most) {
  const int64_t rpc = k > 32 ? 16 : 64;
  const int64_t c = (I + rpc - 1) / rpc;
  return (int)(c < 1 ? 1 : c > most ? most : c);
}

// dynamic shared memory for `rows` rows a CTA
template <int KP>
constexpr size_t mode_smem_bytes(int64_t rows) {
  using S = ModeShape<KP>;
  return ((size_t)rows * S::LDH + (KP == 16 ? (size_t)S::CHUNK * S::LDH : 0) + (size_t)KP * (S::LDG + KP)) *
         sizeof(double);
}
inline size_t mode_smem(int k, int64_t rows) {
  return k <= 16 ? mode_smem_bytes<16>(rows) : k <= 32 ? mode_smem_bytes<32>(rows) : mode_smem_bytes<64>(rows);
}

// 8 bytes to shared memory, asynchronously; zeros (and no access) where !in
__device__ __forceinline__ void mode_copy8(double* dst, const double* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void mode_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void mode_prefetch(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

// sum of the eight warps' values
__device__ __forceinline__ double mode_warp_sums(const double* r) {
  static_assert(MODE_THREADS == 256, "eight warps");
  return ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
}

template <int KP, int UPD>
__device__ __forceinline__ void mode_cluster_body(const ModeArgs& a) {
  using S = ModeShape<KP>;
  constexpr int LPR = S::LPR, CP = S::CP, LDH = S::LDH, CHUNK = S::CHUNK, LDG = S::LDG;
  static_assert(UPD == MODE_NONE || KP == 16, "the fused update is for ranks up to 16");
  cg::cluster_group cluster = cg::this_cluster();
  const int me = (int)cluster.block_rank(), CLm = a.CLm;
  const int k = a.k, kk2 = k * k;
  const int64_t I = a.I;
  extern __shared__ __align__(16) double mode_sm[];
  const int64_t per = (I + CLm - 1) / CLm;
  const int64_t r0 = me < CLm ? (int64_t)me * per : I;
  const int64_t r1 = (r0 + per) < I ? (r0 + per) : I;
  const int nrows = (int)(r1 > r0 ? r1 - r0 : 0);
  double* gs = mode_sm;                    // G of the update at stride LDG; later the factor's U^T U
  double* gsum = gs + KP * LDG;            // U^T U of this CTA's rows
  double* tile = gsum + KP * KP;           // rows at stride LDH
  double* mt = tile + (size_t)per * LDH;   // CHUNK rows of M (update)
  __shared__ double lam[KP];
  __shared__ double red[MODE_THREADS / 32];
  __shared__ double inner_sum;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool err = a.errs != nullptr;

  // e / k for e < 2^16 by one multiplication (the quotient of the rounding
  // error, e / 2^32, stays below 1 / k)
  const uint32_t inv_k = k > 1 ? 0xffffffffu / (uint32_t)k + 1 : 0;
  auto div_k = [&](int e) { return k > 1 ? (int)__umulhi((uint32_t)e, inv_k) : e; };
  // this CTA's slice of the Grams
  const int sl = (kk2 + CLm - 1) / CLm;
  const int s0 = me * sl, s1 = me < CLm ? ((s0 + sl) < kk2 ? (s0 + sl) : kk2) : 0;

  // ---- stage the rows, G and M (columns past k as zeros): every copy is in
  // flight before the first wait
  auto stage = [&](double* dst, const double* src, int rows) {
    for (int e = tid; e < rows * KP; e += MODE_THREADS) {
      const int i = e / KP, c = e % KP;
      mode_copy8(dst + i * LDH + c, src + (c < k ? i * k + c : 0), c < k);
    }
  };
  if (nrows > 0) stage(tile, a.F + r0 * k, nrows);
  if constexpr (UPD != MODE_NONE) {
    for (int e = tid; e < KP * KP; e += MODE_THREADS) {
      const int i = e / KP, j = e % KP;
      const bool in = i < k && j < k;
      mode_copy8(gs + i * LDG + j, a.Gloo + (in ? i * k + j : 0), in);
    }
    if (nrows > 0) stage(mt, a.M + r0 * k, nrows < CHUNK ? nrows : CHUNK);
  }
  // the other modes' Grams and the error's inputs, read at the end (a sector
  // holds four doubles)
  const bool err0 = err && me == 0;
  for (int m = 0; m < a.N && (err0 || a.next >= 0); ++m)
    if (m != a.n)
      for (int e = (err0 ? 0 : s0) + 4 * tid; e < (err0 ? kk2 : s1); e += 4 * MODE_THREADS)
        mode_prefetch(a.Gall + (int64_t)m * kk2 + e);
  if (err0 && tid == 0) {
    mode_prefetch(a.normX2);
    mode_prefetch(a.counter);
  }
  if (UPD == MODE_NONE && err)
    for (int e = 4 * tid; e < nrows * k; e += 4 * MODE_THREADS) mode_prefetch(a.M + r0 * k + e);
  if constexpr (UPD != MODE_NONE) {
    for (int ch = 0; ch < nrows; ch += CHUNK) {
      if (ch > 0) {
        __syncthreads();  // the previous chunk's M is read
        stage(mt, a.M + (r0 + ch) * k, (nrows - ch) < CHUNK ? (nrows - ch) : CHUNK);
      }
      mode_copy_wait();
      __syncthreads();  // M, and for the first chunk G and the rows
      const int q = lane % LPR;
      const int row = ch + warp * S::RPW + lane / LPR;  // this lane's row
      if (ch + warp * S::RPW < nrows) {
        const bool live = row < nrows;
        // lanes past the last row shadow the warp's first one
        double* hrow = tile + (size_t)(live ? row : ch + warp * S::RPW) * LDH;
        // H G of the warp's eight rows, four columns of H a product; a lane's
        // columns are those of its accumulators
        static_assert(LPR == 4, "the accumulators' layout");
        double g[CP / 2][2], h[CP];
#pragma unroll
        for (int p = 0; p < CP / 2; ++p) g[p][0] = g[p][1] = 0.0;
#pragma unroll
        for (int j = 0; j < KP; j += 4)
          if (j < k) {
            const double ha = hrow[j + q];
#pragma unroll
            for (int p = 0; p < CP / 2; ++p)
              dmma_m8n8k4(g[p], ha, gs[(j + q) * LDG + p * 2 * LPR + lane / LPR]);
          }
#pragma unroll
        for (int p = 0; p < CP / 2; ++p) {
          const double2 v = *reinterpret_cast<const double2*>(hrow + p * 2 * LPR + 2 * q);
          h[2 * p] = v.x;
          h[2 * p + 1] = v.y;
        }
        const double* mrow = mt + (size_t)(live ? row - ch : warp * S::RPW) * LDH;
        if constexpr (UPD == MODE_HALS) {
          double m[CP];
#pragma unroll
          for (int p = 0; p < CP / 2; ++p) {
            const double2 v = *reinterpret_cast<const double2*>(mrow + p * 2 * LPR + 2 * q);
            m[2 * p] = v.x;
            m[2 * p + 1] = v.y;
          }
          // columns in order; column i's lane forms the new entry, its
          // change reaches the row's other lanes by one shuffle, and every
          // later column's H G takes it in
#pragma unroll
          for (int p = 0; p < CP / 2; ++p)
#pragma unroll
            for (int o = 0; o < LPR; ++o)
#pragma unroll
              for (int b = 0; b < 2; ++b) {
                const int i = p * 2 * LPR + 2 * o + b;
                if (i < k) {
                  double u = h[2 * p + b] + (m[2 * p + b] - g[p][b]);
                  u = (u < kEps17) ? kEps17 : u;
                  const double delta = __shfl_sync(0xffffffffu, u - h[2 * p + b], o, LPR);
                  if (q == o) h[2 * p + b] = u;
#pragma unroll
                  for (int p2 = p; p2 < CP / 2; ++p2) {
                    const double2 gi = *reinterpret_cast<const double2*>(gs + i * LDG + p2 * 2 * LPR + 2 * q);
                    g[p2][0] = fma(delta, gi.x, g[p2][0]);
                    g[p2][1] = fma(delta, gi.y, g[p2][1]);
                  }
                }
              }
        } else {
#pragma unroll
          for (int p = 0; p < CP / 2; ++p)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
              const int i = p * 2 * LPR + 2 * q + b;
              if (i < k) h[2 * p + b] = (h[2 * p + b] * mrow[i]) / (g[p][b] + a.eps);
            }
        }
        __syncwarp();  // every lane of the row has read the old values
        if (live)
#pragma unroll
          for (int p = 0; p < CP / 2; ++p) {
            const int c = p * 2 * LPR + 2 * q;
            if (c < k) hrow[c] = h[2 * p];
            if (c + 1 < k) hrow[c + 1] = h[2 * p + 1];
          }
        __syncwarp();
      }
    }
  }
  mode_copy_wait();
  __syncthreads();  // the (updated) rows
  if (err) {  // <M, U> over this CTA's rows, a warp's part each
    double inner = 0.0;
    const double* M0 = a.M + r0 * k;
    if (UPD != MODE_NONE && nrows <= CHUNK) {  // M is still in shared memory
      for (int e = tid; e < nrows * k; e += MODE_THREADS) {
        const int i = div_k(e), c = e - i * k;
        inner = fma(mt[i * LDH + c], tile[i * LDH + c], inner);
      }
    } else {
#pragma unroll 4
      for (int e = tid; e < nrows * k; e += MODE_THREADS) {
        const int i = div_k(e), c = e - i * k;
        inner = fma(M0[e], tile[i * LDH + c], inner);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) inner += __shfl_xor_sync(0xffffffffu, inner, o);
    if (lane == 0) red[warp] = inner;
  }

  // ---- U^T U of this CTA's rows: a warp per 8 x 8 block of the upper triangle,
  // four rows a product, in increasing order
  {
    constexpr int KB = S::KB, TPW = S::TPW, NW = MODE_THREADS / 32;
    const int fg = lane >> 2, ft = lane & 3;
    double acc[TPW][2];
    int oa[TPW], ob[TPW];  // columns of the blocks' operands (-1: none)
#pragma unroll
    for (int u = 0; u < TPW; ++u) {
      int ta, tb;
      tri_block(warp + NW * u, KB, ta, tb);
      oa[u] = ta < KB && 8 * ta < k ? 8 * ta : -1;
      ob[u] = 8 * tb;
      acc[u][0] = acc[u][1] = 0.0;
    }
    const double* r = tile + (size_t)ft * LDH + fg;
    auto step = [&](const double* r4, bool in) {
#pragma unroll
      for (int u = 0; u < TPW; ++u)
        if (oa[u] >= 0) dmma_m8n8k4(acc[u], in ? r4[oa[u]] : 0.0, in ? r4[ob[u]] : 0.0);
    };
    int i = 0;
#pragma unroll 4
    for (; i + 4 <= nrows; i += 4) step(r + (size_t)i * LDH, true);
    if (i < nrows) step(r + (size_t)i * LDH, i + ft < nrows);
#pragma unroll
    for (int u = 0; u < TPW; ++u)
      if (oa[u] >= 0) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          gsum[(oa[u] + fg) * KP + ob[u] + 2 * ft + v] = acc[u][v];
          if (oa[u] != ob[u]) gsum[(ob[u] + 2 * ft + v) * KP + oa[u] + fg] = acc[u][v];
        }
      }
    __syncthreads();
    if (err && tid == 0) inner_sum = mode_warp_sums(red);
  }

  // ---- the factor's U^T U in every CTA: partials summed in rank order
  const double* gram = gsum;
  if (cluster.num_blocks() > 1) {
    cluster.sync();
    gram = gs;
    if constexpr (KP == 16) {
      // every CTA reads every partial: few entries, one exchange
      for (int e = tid; e < k * KP && me < CLm; e += MODE_THREADS) {
        double v[MODE_MAX_CL];
#pragma unroll
        for (int b = 0; b < MODE_MAX_CL; ++b) v[b] = b < CLm ? *cluster.map_shared_rank(gsum + e, b) : 0.0;
        double t = v[0];
#pragma unroll
        for (int b = 1; b < MODE_MAX_CL; ++b)
          if (b < CLm) t += v[b];
        gs[e] = t;
      }
      __syncthreads();
    } else {
      // CTA c sums slice c and stores it into every CTA's copy
      const int ne = k * KP, sl = (ne + CLm - 1) / CLm;
      const int e0 = me * sl, e1 = me < CLm ? ((e0 + sl) < ne ? (e0 + sl) : ne) : 0;
      for (int e = e0 + tid; e < e1; e += MODE_THREADS) {
        double v[MODE_MAX_CL];
#pragma unroll
        for (int b = 0; b < MODE_MAX_CL; ++b) v[b] = b < CLm ? *cluster.map_shared_rank(gsum + e, b) : 0.0;
        double t = v[0];
#pragma unroll
        for (int b = 1; b < MODE_MAX_CL; ++b)
          if (b < CLm) t += v[b];
#pragma unroll
        for (int b = 0; b < MODE_MAX_CL; ++b)
          if (b < CLm) *cluster.map_shared_rank(gs + e, b) = t;
      }
      cluster.sync();
    }
  }
  double inner_all = 0.0;
  const bool many = cluster.num_blocks() > 1;
  if (err0 && warp == 0) {
    static_assert(MODE_MAX_CL == 16, "one CTA per lane of a half warp");
    if (lane < CLm) inner_all = *cluster.map_shared_rank(&inner_sum, lane);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) inner_all += __shfl_xor_sync(0xffffffffu, inner_all, o);
  }
  // no CTA reads another's shared memory from here on; a CTA may leave once
  // all have come this far
  if (many) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  if (me < CLm) {
    if (tid < k) lam[tid] = sqrt(gram[tid * KP + tid]);
    __syncthreads();
    // normalised rows
    double* F0 = a.F + r0 * k;
    for (int e = tid; e < nrows * k; e += MODE_THREADS) {
      const int i = div_k(e), c = e - i * k;
      const double nrm = lam[c], u = tile[i * LDH + c];
      F0[e] = nrm > 0 ? u / nrm : u;
    }
    if (me == 0 && tid < k && a.lambda) a.lambda[tid] = lam[tid];
    // G_n and the leave-one-out product of mode `next`: a slice per CTA
    double* Gn = a.Gall + (int64_t)a.n * kk2;
    for (int e = s0 + tid; e < s1; e += MODE_THREADS) {
      const int i = div_k(e), j = e - i * k;
      const double la = lam[i], lb = lam[j], s = gram[i * KP + j];
      const double gn = (la > 0 && lb > 0) ? s / (la * lb) : s;
      Gn[e] = gn;
      if (a.next >= 0) {
        double g = 1.0;
        for (int m = 0; m < a.N; ++m)
          if (m != a.next) g = g * (m == a.n ? gn : a.Gall[(int64_t)m * kk2 + e]);
        a.Gloo[e] = g;
      }
    }
    if (err0) {
      // ||X||^2 - 2 <M, U> + sum_ab lambda_a lambda_b prod_m G_m[a, b], with
      // lambda_a lambda_b G_n[a, b] = (U^T U)_ab
      double mn = 0.0;
      for (int e = tid; e < kk2; e += MODE_THREADS) {
        const int i = div_k(e), j = e - i * k;
        const double la = lam[i], lb = lam[j];
        double g = (la > 0 && lb > 0) ? gram[i * KP + j] : 0.0;
        for (int m = 0; m < a.N; ++m)
          if (m != a.n) g = g * a.Gall[(int64_t)m * kk2 + e];
        mn += g;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mn += __shfl_xor_sync(0xffffffffu, mn, o);
      if (lane == 0) red[warp] = mn;
      __syncthreads();
      if (tid == 0) {
        const double t = mode_warp_sums(red);
        const double nx = *a.normX2;
        const double e2 = nx - 2.0 * inner_all + t;
        const int c = *a.counter;
        a.errs[c] = sqrt(fabs(e2) / nx);
        *a.counter = c + 1;
      }
    }
  }
  if (many) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int KP, int UPD>
__global__ void __launch_bounds__(MODE_THREADS, 1) k_mode_cluster(const __grid_constant__ ModeArgs a) {
  mode_cluster_body<KP, UPD>(a);
}

// Normalisation and Gram of every factor of a context (blockIdx.z = mode; the
// cluster spans the largest factor's CTAs).
struct ModeArgsAll {
  ModeArgs m[kMaxModes];
};
template <int KP>
__global__ void __launch_bounds__(MODE_THREADS) k_mode_all(const __grid_constant__ ModeArgsAll a) {
  mode_cluster_body<KP, MODE_NONE>(a.m[blockIdx.z]);
}

}  // namespace pg
