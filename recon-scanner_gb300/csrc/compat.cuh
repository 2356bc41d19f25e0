// compat.cuh -- the compat-mode cost of a hypothesis (the reference's
// EvaluateCandidate), shared by the compat kernels (compat.cu) and the
// evaluation of given hypotheses (pm.cu).
#pragma once

#include "plane.cuh"

namespace rmvs {

// COMPAT: 1 - mean NCC over valid views (patchmatch_stereo.cpp:344-418), for the
// whole warp: every lane calls it, `have` tells whether this lane has a
// hypothesis.  The lanes take the views in step, so a view's texture is one for
// the warp and the window code may vote.
// `beat`: the caller takes the candidate only below this cost.  NCC is at most
// 1, so after a view the mean over all views is at most (sum + left) / (valid +
// left): once one less that is above `beat` (by more than the sum's rounding)
// the views left cannot change the decision and the lane takes no further
// view; the warp leaves with its last lane.
template <int H, class Ref>
__device__ __forceinline__ HypCost eval_compat_hyp(const Job& J, const PCache& pc, int x, int y, double inv, bool have,
                                                   const RefWindow& rw, const Ref& ref, float* view_cost,
                                                   float beat = kCostInf) {
  bool live = have && !(inv <= 1e-9);
  const double depth = 1.0 / inv;
  live = live && !(depth < J.min_depth || depth > J.max_depth);
  if (view_cost && have && !live)
    for (int s = 0; s < J.num_src; ++s) view_cost[s] = kCostInf;
  const float hi = (float)inv;
  const ff rho{hi, (float)(inv - (double)hi)};
  float sum = 0.f;
  int nvalid = 0;
#pragma unroll 1
  for (int s = 0; s < J.num_src; ++s) {
    if (!__any_sync(0xffffffffu, live)) break;
    ff P[3] = {};
    if (live) pc.get(s, P);
    const ViewResult v = eval_view_compat<H>(J, J.src[s], x, y, P, rho, hi, rw, ref, live);
    if (v.valid) {
      ++nvalid;
      sum += v.ncc;
    }
    if (view_cost && live) view_cost[s] = v.valid ? 1.0f - v.ncc : kCostInf;
    const float left = (float)(J.num_src - 1 - s);
    live = live && !(left > 0.0f && (beat - 1.0f + 1e-5f) * ((float)nvalid + left) < -(sum + left));
  }
  if (!live) return HypCost{kCostInf, 0};
  HypCost r{kCostInf, nvalid};
  if (nvalid == 0) return r;
  float c = 1.0f - sum / (float)nvalid;
  if (c > 3.0f * J.photo_threshold) c = kCostInf;
  r.cost = c;
  return r;
}

// The reference rows a 32 x 4 block of compat pixels reads, in shared memory
// (zeros outside the image: whole windows read none of them).
constexpr int kCompatRows = 4;
template <int H>
struct CompatTile {
  static constexpr int W = 32 + 2 * H, R = kCompatRows + 2 * H;
  float v[H > 0 ? R : 1][H > 0 ? W : 1];
};
template <int H>
struct CompatRef {
  const CompatTile<H>* t;
  int tx, ty;
  __device__ __forceinline__ float operator()(int row, int k) const { return t->v[ty + row][tx + k]; }
};

template <int H>
__device__ __forceinline__ void load_compat_tile(const Job& J, CompatTile<H>& t) {
  if constexpr (H > 0) {
    const int x0 = (int)blockIdx.x * 32 - H, y0 = (int)blockIdx.y * kCompatRows - H;
    for (int i = (int)threadIdx.y * 32 + (int)threadIdx.x; i < t.W * t.R; i += 32 * kCompatRows) {
      const int c = i % t.W, r = i / t.W, xx = x0 + c, yy = y0 + r;
      t.v[r][c] = (xx >= 0 && yy >= 0 && xx < J.w && yy < J.h) ? __ldg(J.ref_box + (size_t)yy * J.w + xx) : 0.0f;
    }
    __syncthreads();
  }
}

}  // namespace rmvs
