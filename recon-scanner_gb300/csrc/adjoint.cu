// adjoint.cu -- the differentiation form: per-hypothesis gradients of the
// aggregated plane cost, and the pose normal equations for pose recovery.
// The math is in adjoint.cuh.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "adjoint.cuh"
#include "kernels.h"

namespace rmvs {

// Per hypothesis: cost, gradient (d, theta, phi), Gauss-Newton matrix (6)
// and, when pose_grad != nullptr, the gradient in every source's pose
// (num_src x 6).  The aggregated cost is the mean of the best_k view costs (the
// search's rule).
//
// A block takes 32 hypotheses; warp w takes the source views w, w + W, ... of
// all of them (W warps), so a few thousand hypotheses fill the chip -- one
// thread per hypothesis left half the schedulers without a warp and the rest
// waiting on one chain of texture reads -- and a warp's lanes read one texture.
// Each view's moments, and after the selection its derivatives, meet in shared
// memory and are added in source order: the sums of the sequential form bit for
// bit.  10^4 hypotheses, 8 sources, 1280x960, 11x11: 1.05 -> 0.28 ms; what is
// left is the latency of one view's two window passes.
constexpr int kAdjHyps = 32;       // hypotheses per block (one warp wide)
constexpr int kAdjMaxWarps = 8;
constexpr int kAdjPerView = 9;     // shared floats per (view, hypothesis): gradient 3, matrix 6

template <int kMode>
__global__ void __launch_bounds__(kAdjHyps * kAdjMaxWarps) k_plane_adjoint(
    Job J, int n, const int* __restrict__ px, const int* __restrict__ py, const double* __restrict__ depth,
    const double* __restrict__ angles, float* cost, float* grad, float* gn, float* pose_grad) {
  extern __shared__ float sh[];
  const int ns = J.num_src, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  float* vc = sh;                                    // [ns][32] view costs, kCostInf invalid
  float* part = sh + (size_t)ns * kAdjHyps;          // [ns][9][32]: first the moments, then the derivatives
  const int i = blockIdx.x * kAdjHyps + lane;
  AdjHyp h;
  const bool ok = i < n && make_adj_hyp(J, px[i], py[i], (float)depth[i], (float)angles[2 * i],
                                        (float)angles[2 * i + 1], &h);
  for (int s = warp; s < ns; s += warps) {
    float c = kCostInf;
    if (ok) {
      const ViewGeo geo = view_geo(J, J.src[s], h);
      const ViewMom mo = view_moments<kMode>(J, J.src[s], geo, h);
      if (mo.valid) c = 1.0f - mo.ncc;
      float* p = part + (size_t)s * kAdjPerView * kAdjHyps + lane;
      p[0 * kAdjHyps] = mo.n;
      p[1 * kAdjHyps] = mo.mr;
      p[2 * kAdjHyps] = mo.ms;
      p[3 * kAdjHyps] = mo.srr;
      p[4 * kAdjHyps] = mo.sss;
      p[5 * kAdjHyps] = mo.srs;
      p[6 * kAdjHyps] = mo.ncc;
    }
    vc[s * kAdjHyps + lane] = c;
  }
  __syncthreads();
  // the k lowest costs, ties to the lower source index (every warp for itself)
  int nvalid = 0;
  for (int s = 0; s < ns; ++s) nvalid += vc[s * kAdjHyps + lane] < kCostInf;
  const int k = (J.best_k <= 0 || J.best_k >= nvalid || J.best_k > kMaxBestK) ? nvalid : J.best_k;
  uint32_t sel = 0;
  float csum = 0.f;
  for (int t = 0; t < k; ++t) {
    int b = -1;
    float cb = kCostInf;
    for (int s = 0; s < ns; ++s) {
      const float c = vc[s * kAdjHyps + lane];
      if (!((sel >> s) & 1u) && c < cb) {
        b = s;
        cb = c;
      }
    }
    sel |= 1u << b;
    csum += cb;
  }
  const float inv_k = 1.0f / (float)max(k, 1);
  for (int s = warp; s < ns; s += warps) {
    float gp[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if ((sel >> s) & 1u) {
      float* p = part + (size_t)s * kAdjPerView * kAdjHyps + lane;  // this thread's own moments
      ViewMom mo;
      mo.n = p[0 * kAdjHyps];
      mo.mr = p[1 * kAdjHyps];
      mo.ms = p[2 * kAdjHyps];
      mo.srr = p[3 * kAdjHyps];
      mo.sss = p[4 * kAdjHyps];
      mo.srs = p[5 * kAdjHyps];
      mo.ncc = p[6 * kAdjHyps];
      mo.valid = true;
      float gs[3], Hs[6], Hp[kPoseH];
      const ViewGeo geo = view_geo(J, J.src[s], h);
      if (pose_grad)
        view_adjoint<kMode, true>(J, J.src[s], geo, h, mo, gs, Hs, gp, Hp);
      else
        view_adjoint<kMode, false>(J, J.src[s], geo, h, mo, gs, Hs, gp, Hp);
      for (int q = 0; q < 3; ++q) p[q * kAdjHyps] = gs[q];
      for (int q = 0; q < 6; ++q) p[(3 + q) * kAdjHyps] = Hs[q];
    }
    if (pose_grad && i < n)
      for (int q = 0; q < 6; ++q) pose_grad[((size_t)i * ns + s) * 6 + q] = gp[q] * inv_k;
  }
  __syncthreads();
  if (i >= n || warp != 0) return;
  float g[3] = {0, 0, 0}, H[6] = {0, 0, 0, 0, 0, 0};
  for (int s = 0; s < ns; ++s) {
    if (!((sel >> s) & 1u)) continue;
    const float* p = part + (size_t)s * kAdjPerView * kAdjHyps + lane;
    for (int q = 0; q < 3; ++q) g[q] += p[q * kAdjHyps] * inv_k;
    for (int q = 0; q < 6; ++q) H[q] += p[(3 + q) * kAdjHyps] * inv_k;
  }
  cost[i] = k > 0 ? csum * inv_k : kCostInf;
  for (int q = 0; q < 3; ++q) grad[3 * i + q] = g[q];
  if (gn)
    for (int q = 0; q < 6; ++q) gn[6 * i + q] = H[q];
}

// Pose normal equations: for every source s, over the given pixels (every
// view valid at a pixel counts, independent of best_k), the sums of the view
// cost c_s, its pose gradient (6) and Gauss-Newton matrix (21), and the
// number of contributing pixels.  One record of kPoseRec floats per (block,
// source); the host adds the blocks in order (deterministic).  The sources are
// the grid's second dimension: they share nothing, and one block walking them
// in turn left most of the chip idle at 10^4 pixels.
constexpr int kPoseRec = 1 + 6 + kPoseH + 1;

template <int kMode>
__global__ void __launch_bounds__(128) k_pose_normal_eq(Job J, int n, const int* __restrict__ px,
                                                        const int* __restrict__ py, const double* __restrict__ depth,
                                                        const double* __restrict__ angles, float* partial) {
  __shared__ float red[4][kPoseRec];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, s = blockIdx.y;
  AdjHyp h;
  const bool ok = i < n && make_adj_hyp(J, px[i], py[i], (float)depth[i], (float)angles[2 * i],
                                        (float)angles[2 * i + 1], &h);
  float rec[kPoseRec];
  for (int k = 0; k < kPoseRec; ++k) rec[k] = 0.f;
  if (ok) {
    const ViewGeo geo = view_geo(J, J.src[s], h);
    const ViewMom mo = view_moments<kMode>(J, J.src[s], geo, h);
    if (mo.valid) {
      float g[3], H[6];
      view_adjoint<kMode, true>(J, J.src[s], geo, h, mo, g, H, rec + 1, rec + 7);
      rec[0] = 1.0f - mo.ncc;
      rec[kPoseRec - 1] = 1.0f;
    }
  }
  // block sum: warp shuffles, then the 4 warps in order
  for (int k = 0; k < kPoseRec; ++k) {
    float v = rec[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < kPoseRec) {
    const int k = threadIdx.x;
    partial[((size_t)blockIdx.x * J.num_src + s) * kPoseRec + k] = ((red[0][k] + red[1][k]) + red[2][k]) + red[3][k];
  }
}

template <class F>
static cudaError_t dispatch_mode(int mode, F&& f) {
  if (mode == kSrcBf16) return f(std::integral_constant<int, kSrcBf16>{});
  return f(std::integral_constant<int, kSrcExact>{});
}

cudaError_t launch_plane_adjoint(const Job& J, int n, const int* px, const int* py, const double* depth,
                                 const double* angles, float* cost, float* grad, float* gn, float* pose_grad,
                                 cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (J.num_src > kMaxSources) return cudaErrorInvalidValue;
  const int warps = J.num_src < kAdjMaxWarps ? J.num_src : kAdjMaxWarps;
  const size_t sm = (size_t)J.num_src * kAdjHyps * (1 + kAdjPerView) * sizeof(float);  // <= 40 KB
  return dispatch_mode(J.src_mode, [&](auto m) {
    k_plane_adjoint<decltype(m)::value><<<(n + kAdjHyps - 1) / kAdjHyps, kAdjHyps * warps, sm, st>>>(
        J, n, px, py, depth, angles, cost, grad, gn, pose_grad);
    return cudaGetLastError();
  });
}

int pose_partial_records() { return kPoseRec; }

cudaError_t launch_pose_normal_eq(const Job& J, int n, const int* px, const int* py, const double* depth,
                                  const double* angles, float* partial, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (J.num_src > kMaxSources) return cudaErrorInvalidValue;
  return dispatch_mode(J.src_mode, [&](auto m) {
    k_pose_normal_eq<decltype(m)::value>
        <<<dim3((n + 127) / 128, J.num_src), 128, 0, st>>>(J, n, px, py, depth, angles, partial);
    return cudaGetLastError();
  });
}

}  // namespace rmvs
