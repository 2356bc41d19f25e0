// plane.cuh -- plane-mode device code shared by the sweep, initialisation and
// refinement kernels: the per-pixel source rays, the cost of
// a hypothesis over its views, the search's candidates, the batch's work items
// and the TMA copy of a reference tile; and the host launchers' helpers.
#pragma once

#include <type_traits>

#include "cost.cuh"
#include "kernels.h"

namespace rmvs {

// ---------------------------------------------------------------------------
// per-thread source-ray cache in shared memory: P[s][c] as float2 (hi, lo)
// ---------------------------------------------------------------------------
struct PCache {
  float2* base;
  int stride;  // threads per block
  int tid;
  __device__ __forceinline__ void get(int s, ff P[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float2 v = base[(s * 3 + c) * stride + tid];
      P[c] = ff{v.x, v.y};
    }
  }
  __device__ __forceinline__ void put(int s, const ff P[3]) const {
#pragma unroll
    for (int c = 0; c < 3; ++c) base[(s * 3 + c) * stride + tid] = make_float2(P[c].hi, P[c].lo);
  }
};

__device__ __forceinline__ void fill_pcache(const Job& J, const PCache& pc, int x, int y, float* rx, float* ry) {
  if (J.hyp && !J.ref_distorted) {
    // plane mode, pinhole reference: the pixel ray and P_s = A_s ray in
    // float-float (~44-bit mantissa) -- no FP64 on the device, whose rate on
    // this part is 1/64 of FP32
    const ff xr = ff_div(ff_add(ff_make((float)x + 0.5f), ff{-J.ffrcx.hi, -J.ffrcx.lo}), J.ffrx);
    const ff yr = ff_div(ff_add(ff_make((float)y + 0.5f), ff{-J.ffrcy.hi, -J.ffrcy.lo}), J.ffry);
    for (int s = 0; s < J.num_src; ++s) {
      const SrcView& S = J.src[s];
      ff P[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) P[i] = ff_add(ff_add(ff_mul(S.Aff[3 * i], xr), ff_mul(S.Aff[3 * i + 1], yr)), S.Aff[3 * i + 2]);
      pc.put(s, P);
    }
    *rx = __fadd_rn(xr.hi, xr.lo);
    *ry = __fadd_rn(yr.hi, yr.lo);
    return;
  }
  double ray[3];
  ref_ray(J, x + 0.5, y + 0.5, ray);
  for (int s = 0; s < J.num_src; ++s) {
    ff P[3];
    source_rays(J, J.src[s], ray, P);
    pc.put(s, P);
  }
  *rx = (float)ray[0];
  *ry = (float)ray[1];
}

// ---------------------------------------------------------------------------
// full hypothesis evaluation over all sources
// ---------------------------------------------------------------------------
struct HypCost {
  float cost;
  int support;
};

__device__ __forceinline__ HypCost finish_plane(float* best, float sum_all, int nvalid, int best_k,
                                                float photo_threshold) {
  HypCost r{kCostInf, nvalid};
  if (nvalid == 0) return r;
  float c;
  if (best_k <= 0 || best_k >= nvalid || best_k > kMaxBestK) {
    c = sum_all / (float)nvalid;
  } else {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < kMaxBestK; ++i)
      if (i < best_k) s += best[i];
    c = s / (float)best_k;
  }
  if (c > 3.0f * photo_threshold) c = kCostInf;
  r.cost = c;
  return r;
}

// The cost of one plane hypothesis from its views: view(s, active) evaluates
// source view s and returns its NCC (valid = -1: not sampled); the cost is
// the mean of the best_k view costs 1 - NCC.  Exact pruning: view costs lie
// in [0, 2], so after each view the final cost is bounded below by letting
// every remaining view be valid at cost 0 -- with K = best_k (or all views),
// n valid so far, r views left and k' = min(K, n + r), cost >= (sum of the
// k' - r lowest costs so far) / k'.  Once that bound is above `beat` (the
// cost a candidate must get below to be taken, with a relative margin that
// covers the rounding of both sums) the remaining views cannot change the
// decision and are not evaluated: the candidate is returned as rejected.
// kCollective: view() is called for every view whatever this lane's state
// (the staged schedule's views are warp-collective), `active` telling it
// whether this lane's hypothesis still needs the view.
template <bool kCollective, class ViewFn>
__device__ __forceinline__ HypCost plane_hyp_cost(const Job& J, bool live, const ViewFn& view, float* view_cost,
                                                  int* counts, float beat) {
  float best[kMaxBestK];
#pragma unroll
  for (int i = 0; i < kMaxBestK; ++i) best[i] = kCostInf;
  float sum_all = 0.f;
  int nvalid = 0;
  const bool all_views = J.best_k <= 0 || J.best_k > kMaxBestK;
  const int K = all_views ? J.num_src : J.best_k;
  const float bar = beat * (1.0f + 4e-6f);
  bool pruned = false;
  for (int s = 0; s < J.num_src; ++s) {
    ViewResult v{0.0f, -1};  // skipped: not sampled
    if (kCollective)
      v = view(s, live && !pruned);
    else if (!pruned)
      v = view(s, true);
    if (counts) counts[1] += v.valid >= 0;
    float c = kCostInf;
    if (v.valid > 0) {
      c = 1.0f - v.ncc;
      ++nvalid;
      sum_all += c;
#pragma unroll
      for (int i = 0; i < kMaxBestK; ++i) {
        const float lo = fminf(best[i], c), hi = fmaxf(best[i], c);
        best[i] = lo;
        c = hi;
      }
      c = 1.0f - v.ncc;
    }
    if (view_cost) view_cost[s] = c;
    const int left = J.num_src - 1 - s;
    if (left > 0 && left < K && nvalid > 0) {
      const int kk = min(K, nvalid + left), j = kk - left;
      float lb;
      if (all_views) {
        lb = sum_all;  // j == nvalid: every valid view so far
      } else {
        lb = 0.f;
#pragma unroll
        for (int i = 0; i < kMaxBestK; ++i)
          if (i < j) lb += best[i];
      }
      pruned = pruned || (j > 0 && lb > bar * (float)kk);
    }
  }
  if (!live || pruned) return HypCost{kCostInf, 0};
  return finish_plane(best, sum_all, nvalid, J.best_k, J.photo_threshold);
}

template <int H, int kMode, class Ref>
__device__ HypCost eval_plane_hyp(const Job& J, const PCache& pc, int x, int y, float rx, float ry, float rho,
                                  float nx, float ny, float nz, const RefWindow& rw, const Ref& ref, float* view_cost,
                                  int* counts = nullptr, float beat = kCostInf) {
  HypCost bad{kCostInf, 0};
  PlaneHyp hp;
  if (!(rho > 0.0f) || rho < J.rho_min || rho > J.rho_max || !make_plane_hyp(J, rx, ry, rho, nx, ny, nz, &hp)) {
    if (view_cost)
      for (int s = 0; s < J.num_src; ++s) view_cost[s] = kCostInf;
    return bad;
  }
  if (counts) ++counts[0];
  return plane_hyp_cost<false>(
      J, true,
      [&](int s, bool) {
        ff P[3];
        pc.get(s, P);
        return eval_view_plane<H, kMode>(J, J.src[s], x, y, P, hp, rw, ref);
      },
      view_cost, counts, beat);
}

// ---------------------------------------------------------------------------
// plane mode
// ---------------------------------------------------------------------------
__device__ __forceinline__ void random_normal(Rng& g, float rx, float ry, float* nx, float* ny, float* nz) {
  // uniform direction, flipped to face the camera, kept off grazing angles
  const float rn = rsqrtf(rx * rx + ry * ry + 1.0f);
  for (int t = 0; t < 8; ++t) {
    const float z = g.sym();
    const float phi = 6.28318530718f * g.uniform();
    const float r = sqrtf(fmaxf(0.f, 1.f - z * z));
    float a = r * __cosf(phi), b = r * __sinf(phi), c = z;
    float d = (a * rx + b * ry + c) * rn;
    if (d > 0.f) {
      a = -a;
      b = -b;
      c = -c;
      d = -d;
    }
    if (d < -0.2f) {
      *nx = a;
      *ny = b;
      *nz = c;
      return;
    }
  }
  *nx = 0.f;
  *ny = 0.f;
  *nz = -1.f;
}

__device__ __forceinline__ void perturb_normal(Rng& g, float rx, float ry, float scale, float* nx, float* ny,
                                               float* nz) {
  float a = *nx + scale * g.sym(), b = *ny + scale * g.sym(), c = *nz + scale * g.sym();
  const float inv = rsqrtf(a * a + b * b + c * c);
  a *= inv;
  b *= inv;
  c *= inv;
  const float rn = rsqrtf(rx * rx + ry * ry + 1.0f);
  if ((a * rx + b * ry + c) * rn < -0.2f) {
    *nx = a;
    *ny = b;
    *nz = c;
  }
}

__device__ __forceinline__ Rng pixel_rng(const Job& J, int idx, int iter, int salt) {
  Rng g;
  g.s = mix64(J.seed ^ ((uint64_t)idx * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)(iter + 1) << 40) ^
              ((uint64_t)salt << 56));
  return g;
}

// ---------------------------------------------------------------------------
// batched plane kernels
// ---------------------------------------------------------------------------
// Every plane-mode run goes through these kernels.  A batch is any set of up
// to kBatchJobs reference views -- uneven sizes and source counts -- that
// share the window size and the interpolation mode.  The batch's job records
// travel in the kernel-parameter (constant) bank: a block reads the record of
// its job with uniform constant loads, which the compiler can re-issue instead
// of holding every field in registers (a copy in shared memory costs the
// unrolled window code hundreds of bytes of spills).  Work items are tiles;
// B.start holds the exclusive prefix of the jobs' tile counts, so an item
// finds its job by a binary search.
__device__ __forceinline__ int find_job(const PlaneBatch& B, int item) {
  int lo = 0, hi = B.njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (B.start[mid] <= item)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Pixel-tile kernels (init, refine, output): one 32 x 4 block per 32 x 4
// pixel tile, grid = the batch's tile count.  Returns the block's job and
// whether this thread's pixel lies inside its image.
__device__ __forceinline__ bool pixel_item(const PlaneBatch& B, int* job, int* x, int* y) {
  const int j = find_job(B, (int)blockIdx.x);
  const int local = (int)blockIdx.x - B.start[j];
  const int tx = (B.jobs[j].w + 31) >> 5;
  *job = j;
  *x = (local % tx) * 32 + (int)threadIdx.x;
  *y = (local / tx) * 4 + (int)threadIdx.y;
  return *x < B.jobs[j].w && *y < B.jobs[j].h;
}

// A neighbour's plane {rho_n at its ray (rxn, ryn), n} carried to the ray
// (rx, ry): the inverse depth at which that ray meets the plane, or -1 when
// the plane does not face the camera along either ray.
__device__ __forceinline__ void plane_candidate_transfer(const float4 hn, float rxn, float ryn, float rx, float ry,
                                                         float* rho) {
  // the neighbour's plane n . X = kappa_n / rho_n, evaluated on this pixel's ray
  const float kn = hn.y * rxn + hn.z * ryn + hn.w;
  const float kp = hn.y * rx + hn.z * ry + hn.w;
  *rho = (kn < 0.f && kp < 0.f) ? hn.x * kp / kn : -1.0f;
}

// A pixel's first plane: random, its parent's at the half-resolution level
// carried to this ray, or its seed cell's depth on a fronto-parallel plane.
__device__ __forceinline__ float4 initial_plane(const Job& J, int x, int y, int idx, float rx, float ry) {
  Rng g = pixel_rng(J, idx, -1, 1);
  float rho = J.rho_min + (J.rho_max - J.rho_min) * g.uniform();
  float nx, ny, nz;
  random_normal(g, rx, ry, &nx, &ny, &nz);
  if (J.coarse_hyp) {
    // the parent's plane at the half-resolution level, carried to this ray
    const int px = min(x >> 1, J.coarse_w - 1), py = min(y >> 1, J.coarse_h - 1);
    const int pi = py * J.coarse_w + px;
    if (J.coarse_cost[pi] < kCostInf) {
      const float4 hn = J.coarse_hyp[pi];
      float rt;
      plane_candidate_transfer(hn, ((float)px + 0.5f - J.crcx) / J.crfx, ((float)py + 0.5f - J.crcy) / J.crfy, rx,
                               ry, &rt);
      if (rt >= J.rho_min && rt <= J.rho_max) {
        rho = rt;
        nx = hn.y;
        ny = hn.z;
        nz = hn.w;
      }
    }
  }
  if (J.seed_depth) {
    const int cx = min(x / 32, J.seed_gx - 1);
    const int cy = y / 32;
    const float sd = J.seed_depth[cy * J.seed_gx + cx];
    if (sd > 0.f) {
      rho = 1.0f / sd;
      nx = 0.f;
      ny = 0.f;
      nz = -1.f;
    }
  }
  return make_float4(rho, nx, ny, nz);
}

// Propagation skips a candidate that is the pixel's current plane: same
// normal bits and an inverse depth within this relative distance (the FP32
// plane transfer through a chain of neighbours rounds at ~1e-7 per step).
constexpr float kSamePlaneRel = 4e-6f;

// Adaptive checkerboard regions (other-colour pixels only: dx + dy odd).
// 4 near "V" regions of 7 pixels and 4 far strips of 11 pixels.
static __constant__ signed char c_near[4][7][2] = {
    {{0, -1}, {-1, -2}, {1, -2}, {-2, -3}, {2, -3}, {-3, -4}, {3, -4}},
    {{0, 1}, {-1, 2}, {1, 2}, {-2, 3}, {2, 3}, {-3, 4}, {3, 4}},
    {{-1, 0}, {-2, -1}, {-2, 1}, {-3, -2}, {-3, 2}, {-4, -3}, {-4, 3}},
    {{1, 0}, {2, -1}, {2, 1}, {3, -2}, {3, 2}, {4, -3}, {4, 3}}};


// Reference-window statistics from the shared tile (same values as
// ref_window for pixels whose window lies inside the image).
template <int H, class Tile>
__device__ __forceinline__ RefWindow tile_window(const Job& J, const Tile& t, int x, int y) {
  RefWindow rw;
  rw.full = x >= H && y >= H && x + H <= J.w - 1 - J.half_pixel && y + H <= J.h - 1 - J.half_pixel;
  if (!rw.full) return ref_window(J, x, y, J.half_pixel);
  float s = 0.f;
#pragma unroll 1
  for (int dy = -H; dy <= H; ++dy) {
    const TileRow r = t.template row<H>(dy);
#pragma unroll
    for (int k = 0; k <= 2 * H; ++k) s += (k & 1) ? r.odd(k >> 1) : r.even(k >> 1);
  }
  rw.mean = s / (float)((2 * H + 1) * (2 * H + 1));
  float q = 0.f;
#pragma unroll 1
  for (int dy = -H; dy <= H; ++dy) {
    const TileRow r = t.template row<H>(dy);
    float qr = 0.f;
#pragma unroll
    for (int k = 0; k <= 2 * H; ++k) {
      const float d = ((k & 1) ? r.odd(k >> 1) : r.even(k >> 1)) - rw.mean;
      qr = fmaf(d, d, qr);
    }
    q += qr;
  }
  rw.sxx = q;
  return rw;
}

// Propagation candidate of region r (0-7) for pixel (x, y): the plane of the
// region's lowest-cost neighbour, carried to this pixel's ray.  False when the
// region offers nothing to learn: no neighbour with a finite cost, the
// current plane again (same normal, inverse depth within rounding of the
// transfer -- in a converged region most regions propose exactly this), or,
// with pruning, the previous region's candidate again (the same plane reached
// through another neighbour: it was rejected, and its cost has not changed).
__device__ __forceinline__ bool propagation_candidate(const Job& J, int x, int y, int r, float rx, float ry,
                                                      float ifx, float ify, const float4& cur, float4& last,
                                                      float4* cand) {
  int best_n = -1;
  float best_c = kCostInf;
  if (r < 4) {
    for (int k = 0; k < 7; ++k) {
      const int nx_ = x + c_near[r][k][0], ny_ = y + c_near[r][k][1];
      if (nx_ < 0 || ny_ < 0 || nx_ >= J.w || ny_ >= J.h) continue;
      const float c = J.cost[ny_ * J.w + nx_];
      if (c < best_c) {
        best_c = c;
        best_n = ny_ * J.w + nx_;
      }
    }
  } else {
    const int d = r - 4;
    const int sx = d == 2 ? -1 : (d == 3 ? 1 : 0);
    const int sy = d == 0 ? -1 : (d == 1 ? 1 : 0);
    for (int k = 0; k < 11; ++k) {
      const int off = 3 + 2 * k;
      const int nx_ = x + sx * off, ny_ = y + sy * off;
      if (nx_ < 0 || ny_ < 0 || nx_ >= J.w || ny_ >= J.h) continue;
      const float c = J.cost[ny_ * J.w + nx_];
      if (c < best_c) {
        best_c = c;
        best_n = ny_ * J.w + nx_;
      }
    }
  }
  if (best_n < 0 || best_c >= kCostInf) return false;
  const float4 hn = J.hyp[best_n];
  const int nxp = best_n % J.w, nyp = best_n / J.w;
  float rho;
  plane_candidate_transfer(hn, ((float)nxp + 0.5f - J.rcx) * ifx, ((float)nyp + 0.5f - J.rcy) * ify, rx, ry, &rho);
  if (!(rho > 0.f)) return false;
  if (hn.y == cur.y && hn.z == cur.z && hn.w == cur.w && fabsf(rho - cur.x) <= kSamePlaneRel * cur.x) return false;
  if (J.prune && hn.y == last.y && hn.z == last.z && hn.w == last.w && rho == last.x) return false;
  last = make_float4(rho, hn.y, hn.z, hn.w);
  *cand = last;
  return true;
}

// Refinement candidate k (0-4) around the current plane `cur`: a random
// plane (k = 0), the inverse depth perturbed (k = 1), the normal perturbed
// (k = 2), both (k = 3) -- ranges shrinking by half per iteration (`scale`)
// -- and the current depth on a fronto-parallel plane (k = 4, the reference's
// model; false when the plane already is one).  The draws are made whether
// or not the candidate is then evaluated (exploring()), so the random stream
// of every pixel is the same under any exploration schedule.
__device__ __forceinline__ bool refinement_candidate(const Job& J, Rng& g, int k, const float4& cur, float rx,
                                                     float ry, float scale, float span, float4* cand) {
  float rho = cur.x, nx = cur.y, ny = cur.z, nz = cur.w;
  if (k == 0) {
    rho = J.rho_min + span * g.uniform();
    random_normal(g, rx, ry, &nx, &ny, &nz);
  } else if (k == 4) {
    if (nx == 0.f && ny == 0.f) return false;
    nx = 0.f;
    ny = 0.f;
    nz = -1.f;
  } else {
    if (k & 1) rho = cur.x + 0.25f * span * scale * g.sym();
    if (k & 2) perturb_normal(g, rx, ry, 0.5f * scale, &nx, &ny, &nz);
  }
  *cand = make_float4(rho, nx, ny, nz);
  return true;
}

// Whether iteration `iter` evaluates refinement candidate k: the exploration
// candidates (k = 0, the random plane; k = 4, the fronto-parallel plane) stop
// at the job's explore_iters -- by then the search has converged and they
// almost never win (at 1920x1440 after coarse-to-fine initialisation: the
// random plane 0.04-0.4 % of its evaluations, the fronto-parallel plane
// 0.2-2.4 %) -- while propagation and the local perturbations go on.
__device__ __forceinline__ bool exploring(const Job& J, int k, int iter) {
  return (k != 0 && k != 4) || J.explore_iters <= 0 || iter < J.explore_iters;
}

// The evaluation counters of a warp into the job's counter (one atomic per
// warp and counter).  Every lane of the warp calls it.
__device__ __forceinline__ void add_counts(const Job& J, const int* counts, int n) {
  for (int i = 0; i < n; ++i) {
    const unsigned int v = __reduce_add_sync(0xffffffffu, (unsigned int)counts[i]);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(J.eval_counter + i, (unsigned long long)v);
  }
}

// ---- TMA staging of the reference tile ----
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// The 3-D box {x, y, z} of `map` into shared memory, completion signalled
// on `bar` (expecting `bytes`).  x is a multiple of 8 floats (32 bytes), y
// may be negative or past the end: TMA fills zeros there.
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar,
                                            uint32_t bytes) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_addr(bar))
      : "memory");
}

// Waits for phase `parity` of `bar`, giving up after `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int limit) {
  for (int i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

constexpr int kTmaWaitPolls = 1 << 22;

// ---------------------------------------------------------------------------
// host side: launch helpers
// ---------------------------------------------------------------------------
inline size_t pcache_bytes(int num_src, int threads) { return (size_t)num_src * 3 * threads * sizeof(float2); }

inline dim3 grid2d(int w, int h, dim3 b) { return dim3((w + b.x - 1) / b.x, (h + b.y - 1) / b.y); }

// Dynamic shared memory above the 48 KB default needs an opt-in per kernel.
template <class K>
inline cudaError_t allow_smem(K* kernel, size_t bytes) {
  if (bytes <= 32 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Calls f(integral_constant<H>, integral_constant<kMode>) for the compiled
// window sizes (11x11, 7x7, and the generic runtime-size path) and source
// modes; BF16 sources have the 11x11 and generic instances only.
template <class F>
inline cudaError_t dispatch_plane(int patch_half, int mode, F&& f) {
  using std::integral_constant;
  if (mode == kSrcTex) {
    if (patch_half == 5) return f(integral_constant<int, 5>{}, integral_constant<int, kSrcTex>{});
    if (patch_half == 3) return f(integral_constant<int, 3>{}, integral_constant<int, kSrcTex>{});
    return f(integral_constant<int, 0>{}, integral_constant<int, kSrcTex>{});
  }
  if (mode == kSrcBf16) {
    if (patch_half == 5) return f(integral_constant<int, 5>{}, integral_constant<int, kSrcBf16>{});
    return f(integral_constant<int, 0>{}, integral_constant<int, kSrcBf16>{});
  }
  if (patch_half == 5) return f(integral_constant<int, 5>{}, integral_constant<int, kSrcExact>{});
  if (patch_half == 3) return f(integral_constant<int, 3>{}, integral_constant<int, kSrcExact>{});
  return f(integral_constant<int, 0>{}, integral_constant<int, kSrcExact>{});
}

}  // namespace rmvs
