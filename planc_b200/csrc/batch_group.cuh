// batch_group.cuh -- grouped launches of a batch of independent factorisations.
//
// One launch runs one phase of the NTF iteration (an update sweep, the
// normalisation + Gram, a multi-TTV, a split-K sum, the error) for every
// member of a batch: blockIdx.z selects the member, whose arguments sit in a
// device table built when the batch's graph is captured. Each member runs
// through the same kernel body, CTA layout and summation order as its own
// launch would (the bodies are shared with the per-context kernels), so a
// grouped run gives the same bits as running the members one by one; the CTAs
// past a member's own grid return at once.
#pragma once
#include "kernels_f64.cuh"
#include "mode_cluster.cuh"

namespace pg {

// HALS / MU sweep of one factor (k_hals_warp / k_mu_warp)
struct GrpUpd {
  double* H;
  const double* M;
  const double* G;
  int64_t I;
  int k;
  unsigned gx;  // the member's own grid
};

template <int KP>
__global__ void __launch_bounds__(256) k_grp_hals(const GrpUpd* __restrict__ a) {
  const GrpUpd& u = a[blockIdx.z];
  if (blockIdx.x >= u.gx) return;
  hals_warp_body<KP>(u.H, u.M, u.G, u.I, u.k, blockIdx.x);
}

template <int KP>
__global__ void __launch_bounds__(256) k_grp_mu(const GrpUpd* __restrict__ a, double eps) {
  const GrpUpd& u = a[blockIdx.z];
  if (blockIdx.x >= u.gx) return;
  mu_warp_body<KP>(u.H, u.M, u.G, u.I, u.k, eps, blockIdx.x);
}

// normalisation + Grams (+ error) of one factor (k_mode_cluster); the launch's
// cluster spans x and has the largest member's size
template <int KP>
__global__ void __launch_bounds__(MODE_THREADS) k_grp_mode(const ModeArgs* __restrict__ a) {
  mode_cluster_body<KP, MODE_NONE>(a[blockIdx.z]);
}

// left multi-TTV of the FP32 intermediate (k_ttv_left<float> / k_ttv_left_f4)
struct GrpTtvL {
  const float* T;
  int64_t A, B;
  int k;
  const double* F;
  double* out;
  unsigned gx;
};

// NB consecutive b a CTA: four where the launch still has CTAs enough (256
// members of 32..256 per mode: 340 us an iteration with one b a CTA, 228 with
// four), one where it would leave SMs idle (the rule is the caller's).
constexpr int GRP_TTVL_NB = 4;
template <int NB>
__global__ void __launch_bounds__(256) k_grp_ttv_left(const GrpTtvL* __restrict__ a) {
  const GrpTtvL& g = a[blockIdx.z];
  if (blockIdx.x >= g.gx) return;
  ttv_left_body<float, NB>(g.T, g.A, g.B, g.k, g.F, g.out, blockIdx.x, g.gx);
}

__global__ void __launch_bounds__(256, 4) k_grp_ttv_left_f4(const GrpTtvL* __restrict__ a) {
  const GrpTtvL& g = a[blockIdx.z];
  if (blockIdx.x >= g.gx) return;
  ttv_left_f4_body(g.T, g.A, g.B, g.k, g.F, g.out, blockIdx.x);
}

// right multi-TTV of the FP32 intermediate (k_ttv_right_tiled<float, KP>)
struct GrpTtvR {
  const float* T;
  int64_t A, B;
  int k;
  WGen wg;
  int64_t bper;
  double* out;
  unsigned gx, gy;
};

template <int KP>
__global__ void __launch_bounds__(256) k_grp_ttv_right(const GrpTtvR* __restrict__ a) {
  const GrpTtvR& g = a[blockIdx.z];
  if (blockIdx.x >= g.gx || blockIdx.y >= g.gy) return;
  ttv_right_tiled_body<float, KP>(g.T, g.A, g.B, g.k, g.wg, g.bper, g.out, blockIdx.x, blockIdx.y);
}

// fixed-order split-K sum (k_reduce_splits_few / k_reduce_splits)
struct GrpRed {
  const double* part;
  int nsplit;
  int64_t stride, n;
  double* out;
  unsigned gx;
};

__global__ void __launch_bounds__(256) k_grp_reduce_few(const GrpRed* __restrict__ a) {
  const GrpRed& g = a[blockIdx.z];
  if (blockIdx.x >= g.gx) return;
  reduce_splits_few_body(g.part, g.nsplit, g.stride, g.n, g.out, blockIdx.x, g.gx);
}

__global__ void k_grp_reduce(const GrpRed* __restrict__ a) {
  const GrpRed& g = a[blockIdx.z];
  if (blockIdx.x >= g.gx) return;
  reduce_splits_body(g.part, g.nsplit, g.stride, g.n, g.out, blockIdx.x, g.gx);
}

// Set-up of a run for every member (blockIdx.z): the error counter at 0 and
// the first leave-one-out product (k_gram_loo); and its results: ne error
// values and the status word, gathered in member order.
struct GrpRun {
  const double* Gall;
  double* Gloo;
  int N, k;
  int* counter;
  const double* errs;
  const int* status;
};

__global__ void __launch_bounds__(256) k_grp_begin(const GrpRun* __restrict__ a) {
  const GrpRun& r = a[blockIdx.z];
  if (threadIdx.x == 0) *r.counter = 0;
  const int kk2 = r.k * r.k;
  for (int e = threadIdx.x; e < kk2; e += 256) {
    double g = 1.0;
    for (int i = 1; i < r.N; ++i) g = g * r.Gall[(int64_t)i * kk2 + e];
    r.Gloo[e] = g;
  }
}

__global__ void __launch_bounds__(256) k_grp_end(const GrpRun* __restrict__ a, int ne,
                                                 double* __restrict__ errs, int* __restrict__ status) {
  const GrpRun& r = a[blockIdx.z];
  for (int e = threadIdx.x; e < ne; e += 256) errs[(int64_t)blockIdx.z * ne + e] = r.errs[e];
  if (threadIdx.x == 0) status[blockIdx.z] = *r.status;
}

}  // namespace pg
