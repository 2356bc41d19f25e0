// split.cu -- the plane-mode kernels for batches too small to fill the chip
// with one thread per pixel: the views of a hypothesis are shared by G warps.
//
// A half-sweep of 160 x 120 has 300 warps for 608 schedulers, and each walks 13
// candidates x 4 views x 121 samples as one chain; of 640 x 480, the last tiles
// to start keep the chip waiting for a third of the launch.  Here G warps own
// the same 32 pixels: each evaluates every G-th source view of every candidate,
// the NCCs meet in shared memory, and all G warps add them up in source order --
// the sums, the selections and the random draws of the one-thread form (pm.cu),
// so the maps are the same bit for bit.  A warp's lanes read one texture, as
// there.  A view cannot be pruned by the views evaluated beside it, so where the
// chip is full anyway the one-thread form does less work: the autotuner times
// both on batches of up to kSplitPixels pixels.  160 x 120, 4 sources, 11 x 11: a
// half-sweep 1.7 -> 0.6 ms, the golden section 1.37 -> 0.34 ms; 640 x 480: 2.5 ->
// 2.1 ms a half-sweep.  Bound by the latency of a warp's chain of samples.
//
// The G warps of a pixel group take the same branches (their state is the same),
// so the named barrier between publishing and reading NCCs is met by all of them.
#include "plane.cuh"

namespace rmvs {

// The NCCs that a pixel group's G warps exchange: two buffers in turn, so that
// one barrier per round is enough (a warp refills a buffer two rounds later,
// behind the barrier that every reader of it has reached).
struct ViewExchange {
  float2* buf;  // [2][G][32]
  int g, G, lane, barrier;
  int turn = 0;
  __device__ __forceinline__ void publish(const ViewResult& v) {
    buf[(turn * G + g) * 32 + lane] = make_float2(v.ncc, (float)v.valid);
    asm volatile("bar.sync %0, %1;" ::"r"(barrier), "r"(32 * G) : "memory");
  }
  __device__ __forceinline__ ViewResult read(int q) const {
    const float2 r = buf[(turn * G + q) * 32 + lane];
    return ViewResult{r.x, (int)r.y};
  }
  __device__ __forceinline__ void next() { turn ^= 1; }
};

// threadIdx.y, which a warp shares (blocks are 32 wide): through a shuffle, so that
// the compiler knows it is uniform and so are the view and its texture handle.
__device__ __forceinline__ int warp_row() { return __shfl_sync(0xffffffffu, (int)threadIdx.y, 0); }

// eval_plane_hyp over a pixel group: `have`, the candidate and `beat` are the
// same in all G warps, and so is the result.
template <int H, int kMode, class Ref>
__device__ __forceinline__ HypCost split_hyp_cost(const Job& J, const PCache& pc, ViewExchange& ex, int x, int y,
                                                  float rx, float ry, const float4& cand, bool have,
                                                  const RefWindow& rw, const Ref& ref, int* counts, float beat) {
  PlaneHyp hp;
  const float rho = cand.x;
  const bool live = have && rho > 0.0f && !(rho < J.rho_min) && !(rho > J.rho_max) &&
                    make_plane_hyp(J, rx, ry, rho, cand.y, cand.z, cand.w, &hp);
  if (!__any_sync(0xffffffffu, live)) return HypCost{kCostInf, 0};
  if (counts) counts[0] += live;
  float best[kMaxBestK];
#pragma unroll
  for (int i = 0; i < kMaxBestK; ++i) best[i] = kCostInf;
  float sum_all = 0.f;
  int nvalid = 0;
  const bool all_views = J.best_k <= 0 || J.best_k > kMaxBestK;
  const int K = all_views ? J.num_src : J.best_k;
  const float bar = beat * (1.0f + 4e-6f);
  bool pruned = false;
#pragma unroll 1
  for (int s0 = 0, k = 0; s0 < J.num_src; s0 += ex.G, ++k) {
    ViewResult mine{0.0f, -1};
    if (live && !pruned && s0 + ex.g < J.num_src) {
      ff P[3];
      pc.get(k, P);
      mine = eval_view_plane<H, kMode>(J, J.src[s0 + ex.g], x, y, P, hp, rw, ref);
    }
    ex.publish(mine);
#pragma unroll 1
    for (int q = 0; q < ex.G && s0 + q < J.num_src; ++q) {
      const ViewResult v = ex.read(q);
      if (counts) counts[1] += v.valid >= 0;
      if (v.valid > 0) {
        float c = 1.0f - v.ncc;
        ++nvalid;
        sum_all += c;
#pragma unroll
        for (int i = 0; i < kMaxBestK; ++i) {
          const float lo = fminf(best[i], c), hi = fmaxf(best[i], c);
          best[i] = lo;
          c = hi;
        }
      }
    }
    ex.next();
    // plane_hyp_cost's bound, over the views of the rounds so far
    const int left = J.num_src - s0 - ex.G;
    if (left > 0 && left < K && nvalid > 0) {
      const int kk = min(K, nvalid + left), j = kk - left;
      float lb = 0.f;
      if (all_views) {
        lb = sum_all;
      } else {
#pragma unroll
        for (int i = 0; i < kMaxBestK; ++i)
          if (i < j) lb += best[i];
      }
      pruned = pruned || (j > 0 && lb > bar * (float)kk);
    }
    if (!__any_sync(0xffffffffu, live && !pruned)) break;
  }
  if (!live || pruned) return HypCost{kCostInf, 0};
  return finish_plane(best, sum_all, nvalid, J.best_k, J.photo_threshold);
}

// One half-sweep: k_plane_sweep's work items (64-column x 2-row tiles), a
// block of 2 pixel groups x G warps per tile.
constexpr int kSplitRows = 2;

template <int H, int kMode>
__global__ void __launch_bounds__(512) k_plane_sweep_split(const __grid_constant__ PlaneBatch B, int total, int* queue,
                                                           int color, int iter) {
  extern __shared__ float2 smem[];
  constexpr int kHalo = H > 0 ? H : 1;
  __shared__ __align__(128) float tile[2 * (kSplitRows + 2 * kHalo) * kTileCols];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_item;
  const int G = (int)blockDim.y / kSplitRows;
  const int nthreads = (int)blockDim.y * 32;
  const int l = (int)threadIdx.x, wy = warp_row(), group = wy % kSplitRows, g = wy / kSplitRows;
  const int tid = (int)threadIdx.y * 32 + l;
  ViewExchange ex{smem + (size_t)group * 2 * G * 32, g, G, l, 1 + group};
  const PCache pc{smem + (size_t)kSplitRows * 2 * G * 32, nthreads, tid};
  // the group's 32 same-colour pixels: 16 column pairs x 2 rows, each quad of
  // lanes 2 x 2 of them (k_plane_sweep)
  const int ty = (l >> 1) & 1, pair = group * 16 + (((l >> 2) << 1) | (l & 1));
  constexpr int box_rows = kSplitRows + 2 * H;
  if constexpr (H > 0) {
    if (tid == 0) mbar_init(&bar, 1);
    __syncthreads();
  }
  uint32_t phase = 0;
  for (;;) {
    if (tid == 0) s_item = atomicAdd(queue, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= total) break;
    const int j = find_job(B, item);
    const Job& J = B.jobs[j];
    const int local = item - B.start[j];
    const int tiles_x = (J.w + 63) >> 6;
    const int bx = local % tiles_x, by = local / tiles_x;
    const int y = by * kSplitRows + ty;
    const int parity = (y + color) & 1;
    const int x = bx * 64 + 2 * pair + parity;
    if constexpr (H > 0) {
      const int polls = B.tma_poll_limit > 0 ? B.tma_poll_limit : kTmaWaitPolls;
      if (tid == 0 && !B.tma_skip)
        tma_load_3d(tile, B.tmaps + j, bx * 32 - 8, by * kSplitRows - H, 0, &bar,
                    (uint32_t)(2 * box_rows * kTileCols * sizeof(float)));
      const bool ok = mbar_wait(&bar, phase, polls);
      phase ^= 1u;
      if (__syncthreads_or(!ok)) {
        // give the copy one more bounded chance to land before leaving
        if (tid == 0) {
          atomicExch(B.err, 1);
          mbar_wait(&bar, phase ^ 1u, polls);
        }
        break;
      }
    }
    const bool inside = x < J.w && y < J.h;
    const int it = iter + J.iter_offset;
    auto sweep = [&](const auto& ref, const RefWindow& rw) {
      const int idx = inside ? y * J.w + x : 0;
      float rx = 0.f, ry = 0.f;
      float4 cur = make_float4(0.f, 0.f, 0.f, 0.f);
      float cur_cost = kCostInf;
      int cur_sup = 0;
      if (inside) {
        fill_pcache(J, pc, x, y, &rx, &ry, g, G);
        cur = J.hyp[idx];
        cur_cost = J.cost[idx];
        cur_sup = J.support[idx];
      }
      const float ifx = 1.0f / J.rfx, ify = 1.0f / J.rfy;
      const float scale = exp2f(-(float)it), span = J.rho_max - J.rho_min;
      int counts[2] = {0, 0};
      float4 last = make_float4(-1.f, 0.f, 0.f, 0.f);
      Rng rng{0};
#pragma unroll 1
      for (int slot = 0; slot < 13; ++slot) {  // 8 propagation regions, 5 refinement candidates
        if (slot == 8) rng = pixel_rng(J, idx, it, 2 + color);
        float4 cand = make_float4(0.f, 0.f, 0.f, 0.f);
        const bool have =
            inside && (slot < 8 ? propagation_candidate(J, x, y, slot, rx, ry, ifx, ify, cur, last, &cand)
                                : refinement_candidate(J, rng, slot - 8, cur, rx, ry, scale, span, &cand) &&
                                      exploring(J, slot - 8, it));
        const HypCost c = split_hyp_cost<H, kMode>(J, pc, ex, x, y, rx, ry, cand, have, rw, ref, counts,
                                                   J.prune ? cur_cost : kCostInf);
        if (have && c.cost < cur_cost) {
          cur_cost = c.cost;
          cur = cand;
          cur_sup = c.support;
        }
      }
      if (g == 0) {  // the other warps hold the same
        if (J.eval_counter) add_counts(J, 0xffffffffu, counts, 2);
        if (inside) {
          J.hyp[idx] = cur;
          J.cost[idx] = cur_cost;
          J.support[idx] = (uint8_t)min(cur_sup, 255);
        }
      }
    };
    RefWindow rw{0.0f, 0.0f, false};
    if constexpr (H > 0) {
      const float* plane0 = tile;
      const float* plane1 = tile + box_rows * kTileCols;
      const TileRef<4> ref{parity ? plane1 : plane0, parity ? plane0 : plane1, pair, parity, ty};
      if (inside) rw = tile_window<H>(J, ref, x, y);
      sweep(ref, rw);
    } else {
      const GlobalRef<4> ref{J.pref, J.w, x, y};
      if (inside) rw = ref_window(J, x, y, J.half_pixel);
      sweep(ref, rw);
    }
    __syncthreads();
  }
}

// k_plane_init over pixel groups: a 32 x 4 pixel tile per block, 4 groups of G
// warps.
template <int H, int kMode>
__global__ void __launch_bounds__(512) k_plane_init_split(const __grid_constant__ PlaneBatch B, int* queues,
                                                          int num_queues) {
  extern __shared__ float2 smem[];
  const int G = (int)blockDim.y / 4, nthreads = (int)blockDim.y * 32;
  const int l = (int)threadIdx.x, wy = warp_row(), group = wy & 3, g = wy >> 2;
  const int tid = (int)threadIdx.y * 32 + l;
  if (blockIdx.x == 0)
    for (int q = tid; q < num_queues; q += nthreads) queues[q] = 0;
  const int j = find_job(B, (int)blockIdx.x);
  const Job& J = B.jobs[j];
  const int local = (int)blockIdx.x - B.start[j], tx = (J.w + 31) >> 5;
  const int x = (local % tx) * 32 + l, y = (local / tx) * 4 + group;
  const bool inside = x < J.w && y < J.h;
  ViewExchange ex{smem + (size_t)group * 2 * G * 32, g, G, l, 1 + group};
  const PCache pc{smem + (size_t)4 * 2 * G * 32, nthreads, tid};
  const int idx = inside ? y * J.w + x : 0;
  float rx = 0.f, ry = 0.f;
  float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
  RefWindow rw{0.0f, 0.0f, false};
  if (inside) {
    if (idx == 0 && g == 0) *J.out_filled = 0u;
    fill_pcache(J, pc, x, y, &rx, &ry, g, G);
    h = initial_plane(J, x, y, idx, rx, ry);
    rw = ref_window(J, x, y, J.half_pixel);
  }
  const GlobalRef<4> ref{J.pref, J.w, x, y};
  const HypCost c =
      split_hyp_cost<H, kMode>(J, pc, ex, x, y, rx, ry, h, inside, rw, ref, static_cast<int*>(nullptr), kCostInf);
  if (inside && g == 0) {
    J.hyp[idx] = h;
    J.cost[idx] = c.cost;
    J.support[idx] = (uint8_t)min(c.support, 255);
  }
}

// k_plane_refine (golden section) over pixel groups.
template <int H, int kMode>
__global__ void __launch_bounds__(512) k_plane_refine_split(const __grid_constant__ PlaneBatch B) {
  extern __shared__ float2 smem[];
  const int G = (int)blockDim.y / 4, nthreads = (int)blockDim.y * 32;
  const int l = (int)threadIdx.x, wy = warp_row(), group = wy & 3, g = wy >> 2;
  const int j = find_job(B, (int)blockIdx.x);
  const Job& J = B.jobs[j];
  if (J.refine_iters <= 0 || J.refine_mode != 1) return;
  const int local = (int)blockIdx.x - B.start[j], tx = (J.w + 31) >> 5;
  const int x = (local % tx) * 32 + l, y = (local / tx) * 4 + group;
  ViewExchange ex{smem + (size_t)group * 2 * G * 32, g, G, l, 1 + group};
  const PCache pc{smem + (size_t)4 * 2 * G * 32, nthreads, (int)threadIdx.y * 32 + l};
  bool inside = x < J.w && y < J.h;
  const int idx = inside ? y * J.w + x : 0;
  float4 h0 = make_float4(0.f, 0.f, 0.f, 0.f);
  float best_c = kCostInf;
  int best_s = 0;
  if (inside) {
    h0 = J.hyp[idx];
    best_c = J.cost[idx];
    best_s = J.support[idx];
  }
  inside = inside && best_c < 1e29f;
  float rx = 0.f, ry = 0.f;
  RefWindow rw{0.0f, 0.0f, false};
  if (inside) {
    fill_pcache(J, pc, x, y, &rx, &ry, g, G);
    rw = ref_window(J, x, y, J.half_pixel);
  }
  const GlobalRef<4> ref{J.pref, J.w, x, y};
  float best_d = h0.x;
  float lo = fmaxf(J.rho_min, best_d - J.inv_per_px);
  float hi = fminf(J.rho_max, best_d + J.inv_per_px);
  const bool section = inside && hi > lo;
  const float inv_phi = 0.618033988749895f;
  float c1 = hi - inv_phi * (hi - lo), c2 = lo + inv_phi * (hi - lo);
  HypCost f1{kCostInf, 0}, f2{kCostInf, 0};
#pragma unroll 1
  for (int t = 0; t <= J.refine_iters + 2; ++t) {  // both first points, the iterations, the midpoint
    float v;
    bool left = t == 0;
    if (t == 0) {
      v = c1;
    } else if (t == 1) {
      v = c2;
    } else if (t < J.refine_iters + 2) {
      left = f1.cost < f2.cost;
      if (left) {
        hi = c2;
        c2 = c1;
        f2 = f1;
        v = c1 = hi - inv_phi * (hi - lo);
      } else {
        lo = c1;
        c1 = c2;
        f1 = f2;
        v = c2 = lo + inv_phi * (hi - lo);
      }
    } else {
      v = 0.5f * (lo + hi);
    }
    const HypCost f = split_hyp_cost<H, kMode>(J, pc, ex, x, y, rx, ry, make_float4(v, h0.y, h0.z, h0.w), section, rw,
                                               ref, static_cast<int*>(nullptr), kCostInf);
    if (t == J.refine_iters + 2) {
      if (f.cost < best_c) {
        best_c = f.cost;
        best_d = v;
        best_s = f.support;
      }
    } else if (left) {
      f1 = f;
    } else {
      f2 = f;
    }
  }
  if (section) {
    if (f1.cost < best_c) {
      best_c = f1.cost;
      best_d = c1;
      best_s = f1.support;
    }
    if (f2.cost < best_c) {
      best_c = f2.cost;
      best_d = c2;
      best_s = f2.support;
    }
  }
  if (inside && g == 0) {
    J.hyp[idx] = make_float4(best_d, h0.y, h0.z, h0.w);
    J.cost[idx] = best_c;
    J.support[idx] = (uint8_t)min(best_s, 255);
  }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// The groups' exchange buffers, then the source rays of each warp's own views.
static size_t split_smem_bytes(int max_src, int groups, int G) {
  return (size_t)groups * 2 * G * 32 * sizeof(float2) + pcache_bytes((max_src + G - 1) / G, groups * G * 32);
}

cudaError_t plane_split_occupancy(int patch_half, int mode, int max_src, int G, int* blocks_per_sm) {
  const size_t sm = split_smem_bytes(max_src, kSplitRows, G);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_sweep_split<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, 32 * kSplitRows * G, sm);
  });
}

cudaError_t launch_plane_sweep_split(const PlaneBatch& B, int total, int* queue, int patch_half, int mode, int max_src,
                                     int G, int grid, int color, int iter, cudaStream_t st) {
  if (total <= 0) return cudaSuccess;
  if (G < 2 || G > kMaxSplit || grid < 1 || total > B.start[B.njobs]) return cudaErrorInvalidValue;
  const size_t sm = split_smem_bytes(max_src, kSplitRows, G);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_sweep_split<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<grid, dim3(32, kSplitRows * G), sm, st>>>(B, total, queue, color, iter);
    return cudaGetLastError();
  });
}

// The pixel-tile kernels have 4 groups a block: at most 4 warps each.
static int tile_split(int G) { return G < 4 ? G : 4; }

cudaError_t launch_plane_init_split(const PlaneBatch& B, int patch_half, int mode, int max_src, int G, int* queues,
                                    int num_queues, cudaStream_t st) {
  const int total = B.start[B.njobs];
  if (total <= 0) return cudaSuccess;
  G = tile_split(G);
  const size_t sm = split_smem_bytes(max_src, 4, G);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_init_split<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<total, dim3(32, 4 * G), sm, st>>>(B, queues, num_queues);
    return cudaGetLastError();
  });
}

cudaError_t launch_plane_refine_split(const PlaneBatch& B, int patch_half, int mode, int max_src, int G,
                                      cudaStream_t st) {
  const int total = B.start[B.njobs];
  if (total <= 0) return cudaSuccess;
  G = tile_split(G);
  const size_t sm = split_smem_bytes(max_src, 4, G);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_refine_split<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<total, dim3(32, 4 * G), sm, st>>>(B);
    return cudaGetLastError();
  });
}

}  // namespace rmvs
