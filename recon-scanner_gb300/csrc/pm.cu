// pm.cu -- PatchMatch kernels: hypothesis evaluation, plane-mode red-black
// sweeps, outputs, refinement (compat mode: compat.cu).
//
// Plane mode (the GB300 engine): per-pixel plane hypotheses (inverse depth,
// normal), red-black checkerboard propagation -- a half-sweep updates one
// colour reading only the other colour, so it is race-free and
// deterministic -- with adaptive neighbour selection (best cost in each of 8
// regions) and random perturbation; cost = mean of the best_k view costs.
// Work that cannot change a pixel's fate is skipped (a propagation candidate
// equal to the one just rejected; the remaining source windows of a
// candidate once its best-k bound rules it out): the maps do not depend on
// it, and Job::prune = 0 turns it off.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "adjoint.cuh"
#include "kernels.h"
#include "plane.cuh"

namespace rmvs {

// ---------------------------------------------------------------------------
// batch evaluation of given plane hypotheses (parity instrument, adjoint driver)
// ---------------------------------------------------------------------------
template <int H, int kMode>
__global__ void __launch_bounds__(128, 4) k_eval_hyps(Job J, int n, const int* __restrict__ px,
                                                      const int* __restrict__ py, const double* __restrict__ inv,
                                                      const float* __restrict__ normals, float* out_cost,
                                                      int* out_support, float* out_view_cost) {
  extern __shared__ float2 smem[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  PCache pc{smem, (int)blockDim.x, (int)threadIdx.x};
  if (i >= n) return;
  const int x = px[i], y = py[i];
  float rx, ry;
  fill_pcache(J, pc, x, y, &rx, &ry);
  float* vc = out_view_cost ? out_view_cost + (size_t)i * J.num_src : nullptr;
  const RefWindow rw = ref_window(J, x, y, J.half_pixel);
  const GlobalRef<> ref{J.pref, J.w, x, y};
  const HypCost r = eval_plane_hyp<H, kMode>(J, pc, x, y, rx, ry, (float)inv[i], normals[3 * i], normals[3 * i + 1],
                                             normals[3 * i + 2], rw, ref, vc);
  out_cost[i] = r.cost;
  out_support[i] = r.support;
}

// Random initialisation (and seed cells) + initial cost.  Block 0 also zeroes
// the work counters of the persistent sweeps that follow, and each job's
// first pixel zeroes its filled counter.
template <int H, int kMode>
__global__ void __launch_bounds__(128, 4) k_plane_init(const __grid_constant__ PlaneBatch B, int* queues,
                                                       int num_queues) {
  extern __shared__ float2 smem[];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  if (blockIdx.x == 0)
    for (int q = tid; q < num_queues; q += 128) queues[q] = 0;
  int j, x, y;
  if (!pixel_item(B, &j, &x, &y)) return;
  const Job& J = B.jobs[j];
  PCache pc{smem, 128, tid};
  const int idx = y * J.w + x;
  if (idx == 0) *J.out_filled = 0u;
  float rx, ry;
  fill_pcache(J, pc, x, y, &rx, &ry);
  const float4 h = initial_plane(J, x, y, idx, rx, ry);
  const RefWindow rw = ref_window(J, x, y, J.half_pixel);
  const GlobalRef<> ref{J.pref, J.w, x, y};
  const HypCost c = eval_plane_hyp<H, kMode>(J, pc, x, y, rx, ry, h.x, h.y, h.z, h.w, rw, ref, nullptr);
  J.hyp[idx] = h;
  J.cost[idx] = c.cost;
  J.support[idx] = (uint8_t)min(c.support, 255);
}

// The same value, which the compiler may not have computed earlier: what
// follows from it is computed where it stands.  In the texture-read sweep's slot
// loop that takes the spill stack from 120 to 64 bytes a thread (texture results
// and spills come through the same pipe): with the tile's two row pointers in
// place of five values, 2 maps of 1920x1440 with 8 sources 448 -> 425 ms whole, a
// mixed batch of four 179 -> 167 ms, a stage of nine 640x480 maps 79 -> 74 ms.
__device__ __forceinline__ int again(int v) {
  asm volatile("" : "+r"(v));
  return v;
}
__device__ __forceinline__ float again(float v) {
  asm volatile("" : "+f"(v));
  return v;
}

// One red-black half-sweep of one pixel: propagation from the best-cost
// neighbour of each of the 8 adaptive regions, then 5 refinement hypotheses.
// Adds to `counts`: hypotheses evaluated, source windows sampled.
template <int H, int kMode, class RefT>
__device__ __forceinline__ void sweep_pixel(const Job& J, const PCache& pc, const RefT& ref, const RefWindow& rw,
                                            int x, int y, int color, int iter, int* counts) {
  int idx = y * J.w + x;
  float rx, ry;
  fill_pcache(J, pc, x, y, &rx, &ry);
  float4 cur = J.hyp[idx];
  float cur_cost = J.cost[idx];
  int cur_sup = J.support[idx];

  float4 last = make_float4(-1.f, 0.f, 0.f, 0.f);  // the last candidate evaluated
  Rng g{0};
  // slots 0-7: propagation regions; 8-12: refinement candidates -- one loop, so
  // that the window code is compiled once: with a copy per half, warps waited
  // for instructions (exact reads, a batch of four maps: 186 -> 159 ms over 8
  // half-sweeps; texture-unit reads, bound by that unit, gain 12 % at the
  // half-resolution level and lose 1.5 % at 1920x1440)
#pragma unroll 1
  for (int slot = 0; slot < 13; ++slot) {
    // what the window code has no use for is computed again for each slot
    // (`again`), not kept in the 96 registers across it
    const int it = again(iter);
    if (slot == 8) g = pixel_rng(J, again(y) * J.w + x, it, 2 + color);
    const float scale = exp2f(-(float)it);  // 1, 1/2, 1/4, ...
    const float span = again(J.rho_max) - J.rho_min;
    const float ifx = 1.0f / again(J.rfx), ify = 1.0f / again(J.rfy);
    float4 cand;
    if (!(slot < 8 ? propagation_candidate(J, x, y, slot, rx, ry, ifx, ify, cur, last, &cand)
                   : refinement_candidate(J, g, slot - 8, cur, rx, ry, scale, span, &cand) &&
                         exploring(J, slot - 8, it)))
      continue;
    const HypCost c = eval_plane_hyp<H, kMode>(J, pc, x, y, rx, ry, cand.x, cand.y, cand.z, cand.w, rw, ref, nullptr,
                                               counts, J.prune ? cur_cost : kCostInf);
    if (c.cost < cur_cost) {
      cur_cost = c.cost;
      cur = cand;
      cur_sup = c.support;
    }
  }
  idx = again(y) * J.w + x;
  J.hyp[idx] = cur;
  J.cost[idx] = cur_cost;
  J.support[idx] = (uint8_t)min(cur_sup, 255);
}

// ---- the staged-window schedule ----
// The 2-D box {x, y} of `map` (a tensor map in global memory) into shared
// memory, completion signalled on `bar`.  x is even (8-byte elements:
// 16-byte aligned rows); x or y may be negative or past the end (zeros).
__device__ __forceinline__ void tma_load_2d(void* dst, const void* map, int x, int y, uint64_t* bar,
                                            uint32_t bytes) {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar))
      : "memory");
}

// One warp's source box and its copy state (the same in every lane).
struct WarpBox {
  float2* box;     // kStageH rows x kStageW texel pairs, 128-byte aligned
  uint64_t* bar;   // the box's mbarrier (arrival count 1)
  uint32_t phase;  // parity of the next copy's completion
  int polls;       // wait limit
  int* err;        // set when a wait runs out
  bool dead;       // a wait ran out: no further copies into this box in this launch
};

// One source view of one candidate for the whole warp (every lane calls it;
// `act`: this lane's hypothesis is live for the view).  The lanes whose
// windows lie fully inside the source (the fast path) pool the texels they
// read -- the corners' footprints with a margin of one texel for rounding --
// into one box; when it fits kStageW x kStageH, lane 0 copies it from the
// view's pair image by TMA and every lane waits (bounded) for it, then those
// windows are read from shared memory.  Other windows, and full ones whose
// box does not fit, read the texture.  Either way a window's NCC is the same
// bit for bit.
template <int H, class Ref>
__device__ __forceinline__ ViewResult eval_view_staged(const Job& J, const SrcView& S, int x, int y, const ff P[3],
                                                       const PlaneHyp& hp, bool act, const RefWindow& rw,
                                                       const Ref& ref, WarpBox& wb, int* counts) {
  WindowPlace g;
  const bool geo = act && place_window<H>(J, S, P, hp, rw, &g);
  int x0 = 0x7fffffff, x1 = (int)0x80000000, y0 = 0x7fffffff, y1 = (int)0x80000000;
  if (geo && g.full) {
    // footprints of index coordinates in [min, max]: texels floor(min) - 1 ..
    // floor(max) + 1 (an exact tie reads one texel lower), plus the margin
    x0 = g.iu + (int)floorf(g.umin) - 2;
    x1 = g.iu + (int)floorf(g.umax) + 2;
    y0 = g.iv + (int)floorf(g.vmin) - 2;
    y1 = g.iv + (int)floorf(g.vmax) + 2;
  }
  x0 = __reduce_min_sync(0xffffffffu, x0);
  x1 = __reduce_max_sync(0xffffffffu, x1);
  y0 = __reduce_min_sync(0xffffffffu, y0);
  y1 = __reduce_max_sync(0xffffffffu, y1);
  const int ax = x0 & ~1;  // an even first pair: 16-byte TMA rows
  // pair element e of a box row holds texels ax + e and ax + e + 1, so the
  // texels ax .. x1 need x1 - ax <= kStageW; rows y0 .. y1 need kStageH
  bool staged = S.pair_map != nullptr && !wb.dead && x0 <= x1 && x1 - ax <= kStageW && y1 - y0 < kStageH;
  if (staged) {
    if ((threadIdx.x & 31) == 0) tma_load_2d(wb.box, S.pair_map, ax, y0, wb.bar, (uint32_t)kStageBytes);
    const bool ok = __all_sync(0xffffffffu, mbar_wait(wb.bar, wb.phase, wb.polls));
    wb.phase ^= 1u;
    if (!ok) {
      // the copy may still land: the box is not used again in this launch
      wb.dead = true;
      staged = false;
      if ((threadIdx.x & 31) == 0) atomicExch(wb.err, 1);
    }
  }
  ViewResult v{0.0f, -1};
  if (geo) {
    if (staged && g.full) {
      v = eval_view_box<H>(J, g, rw, ref, wb.box, ax, y0);
      ++counts[2];
    } else {
      v = eval_view_placed<H, kSrcExact>(J, S, x, y, g, hp, rw, ref);
    }
  }
  __syncwarp();  // every lane is done with the box before the next copy into it
  return v;
}

// eval_plane_hyp for the staged schedule: the view loop runs in step across
// the warp (J is the same for the whole block); `have` = this lane has a
// candidate in this slot.
template <int H, class Ref>
__device__ __forceinline__ HypCost eval_plane_hyp_staged(const Job& J, const PCache& pc, int x, int y, float rx,
                                                         float ry, const float4& cand, bool have, const RefWindow& rw,
                                                         const Ref& ref, int* counts, float beat, WarpBox& wb) {
  PlaneHyp hp;
  const float rho = cand.x;
  const bool live = have && rho > 0.0f && !(rho < J.rho_min) && !(rho > J.rho_max) &&
                    make_plane_hyp(J, rx, ry, rho, cand.y, cand.z, cand.w, &hp);
  if (live) ++counts[0];
  return plane_hyp_cost<true>(
      J, live,
      [&](int s, bool act) {
        ff P[3] = {};
        if (act) pc.get(s, P);
        return eval_view_staged<H>(J, J.src[s], x, y, P, hp, act, rw, ref, wb, counts);
      },
      nullptr, counts, beat);
}

// sweep_pixel for the staged schedule: every lane of the warp runs every
// candidate slot and view in step; a lane outside the image, or without a
// candidate in a slot, only takes part in the warp's collective steps.
template <int H, class RefT>
__device__ __forceinline__ void sweep_pixel_staged(const Job& J, const PCache& pc, const RefT& ref, bool inside,
                                                   int x, int y, int color, int iter, WarpBox& wb) {
  const int idx = inside ? y * J.w + x : 0;
  RefWindow rw{0.0f, 0.0f, false};
  float rx = 0.f, ry = 0.f;
  float4 cur = make_float4(0.f, 0.f, 0.f, 0.f);
  float cur_cost = kCostInf;
  int cur_sup = 0;
  if (inside) {
    rw = tile_window<H>(J, ref, x, y);
    fill_pcache(J, pc, x, y, &rx, &ry);
    cur = J.hyp[idx];
    cur_cost = J.cost[idx];
    cur_sup = J.support[idx];
  }
  const float ifx = 1.0f / J.rfx, ify = 1.0f / J.rfy;
  int counts[3] = {0, 0, 0};  // hypotheses, source windows sampled, of them read from a staged box
  float4 last = make_float4(-1.f, 0.f, 0.f, 0.f);
  Rng g{0};
  const float scale = exp2f(-(float)iter);
  const float span = J.rho_max - J.rho_min;
  // slots 0-7: propagation regions; 8-12: refinement candidates (one loop,
  // so that the hypothesis evaluation is instantiated once)
  for (int slot = 0; slot < 13; ++slot) {
    if (slot == 8) g = pixel_rng(J, idx, iter, 2 + color);
    float4 cand = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool have =
        inside && (slot < 8 ? propagation_candidate(J, x, y, slot, rx, ry, ifx, ify, cur, last, &cand)
                            : refinement_candidate(J, g, slot - 8, cur, rx, ry, scale, span, &cand) &&
                                  exploring(J, slot - 8, iter));
    const HypCost c = eval_plane_hyp_staged<H>(J, pc, x, y, rx, ry, cand, have, rw, ref, counts,
                                               J.prune ? cur_cost : kCostInf, wb);
    if (have && c.cost < cur_cost) {
      cur_cost = c.cost;
      cur = cand;
      cur_sup = c.support;
    }
  }
  if (J.eval_counter) add_counts(J, counts, 3);
  if (inside) {
    J.hyp[idx] = cur;
    J.cost[idx] = cur_cost;
    J.support[idx] = (uint8_t)min(cur_sup, 255);
  }
}

// One red-black half-sweep over a whole batch: a persistent kernel (grid =
// resident blocks) whose blocks pull work items -- 64-column x R-row tiles,
// R = blockDim.y -- from an atomic counter until the batch is exhausted.  A
// block of 32 x R threads owns the 32 same-colour pixels of each of its R
// rows; the reference rows the tile reads (R + 2H rows, the 64 columns, 16
// more on the left and 32 on the right) are staged once into shared memory as
// even / odd column planes from the de-interleaved reference copy.
//
// A warp owns a compact patch, not a row: RW = min(R, 4) rows x 32 / RW
// same-colour pixels (16 x 4 pixels for R >= 4).  Each window sample of a
// warp is one texture instruction over its 32 pixels, and their source
// footprints then cluster in a 2-D patch of the source instead of spreading
// along a 64-pixel row: fewer texture-cache lines per instruction.  `queue`
// is this launch's work counter (zeroed by the init kernel); `total` its item
// count -- jobs with fewer iterations than `iter + 1` sit at the end of the
// job order and fall outside it.
//
// kStaged (exact interpolation, H > 0): the staged-window schedule -- each
// warp owns a kStageW x kStageH box of texel pairs at the start of the
// dynamic shared memory (the source-ray cache follows it) and reads the
// windows its pixels share from there (eval_view_staged).
//
// kCut: the group of reads in windows of a size without an instance
// (plane_window).
template <int H, int kMode, bool kStaged, int kCut = 4>
__global__ void __maxnreg__(kStaged ? 128 : 96) k_plane_sweep(const __grid_constant__ PlaneBatch B, int total, int* queue, int color,
                                              int iter) {
  static_assert(!kStaged || (H > 0 && kMode == kSrcExact), "the staged schedule reads exact 2x2 footprints");
  extern __shared__ float2 smem[];
  constexpr int kHalo = H > 0 ? H : 1;
  __shared__ __align__(128) float tile[2 * (kMaxTileRows + 2 * kHalo) * kTileCols];
  __shared__ __align__(8) uint64_t bar;
  __shared__ __align__(8) uint64_t box_bar[kStaged ? kMaxTileRows : 1];
  __shared__ int s_item;
  const int R = (int)blockDim.y;
  const int nthreads = 32 * R;
  const int tid = threadIdx.y * 32 + threadIdx.x;
  float2* pc_base = smem;
  WarpBox wb{nullptr, nullptr, 0u, 0, B.err, false};
  if constexpr (kStaged) {
    // the boxes first, from the first 128-byte boundary (TMA destinations)
    const uint32_t a = smem_addr(smem);
    char* boxes = reinterpret_cast<char*>(smem) + (((a + 127u) & ~127u) - a);
    wb.box = reinterpret_cast<float2*>(boxes + (size_t)threadIdx.y * kStageBytes);
    wb.bar = &box_bar[threadIdx.y];
    wb.polls = B.tma_poll_limit > 0 ? B.tma_poll_limit : kTmaWaitPolls;
    pc_base = reinterpret_cast<float2*>(boxes + (size_t)R * kStageBytes);
    if (threadIdx.x == 0) mbar_init(wb.bar, 1);
  }
  const PCache pc{pc_base, nthreads, tid};
  const int box_rows = R + 2 * H;
  // this thread's pixel in the tile: row ty, same-colour column pair `pair`.
  // A warp covers RW rows x PW pairs; within it each quad of lanes (the
  // texture unit's unit of work) takes 2 rows x 2 pairs -- a compact 4 x 2
  // pixel diamond whose source footprints share texture-cache sectors --
  // rather than 4 pairs of one row.
  const int RW = R < 4 ? R : 4;        // rows per warp
  const int PW = 32 / RW;              // pixels per warp row
  const int w = (int)threadIdx.y, l = (int)threadIdx.x;
  int r_in, c_in;
  if (RW == 4) {
    r_in = ((l >> 4) << 1) | ((l >> 1) & 1);
    c_in = (((l >> 2) & 3) << 1) | (l & 1);
  } else if (RW == 2) {
    r_in = (l >> 1) & 1;
    c_in = ((l >> 2) << 1) | (l & 1);
  } else {
    r_in = 0;
    c_in = l;
  }
  const int ty = (w / RW) * RW + r_in;
  const int pair = (w % RW) * PW + c_in;
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
    const int y = by * R + ty;
    const int parity = (y + color) & 1;
    const int x = bx * 64 + 2 * pair + parity;
    if constexpr (H > 0) {
      // the tile: planes [2][box_rows][kTileCols] of ref_de from column bx*32 - 8 and
      // row by*R - H, one TMA box (zeros outside the image)
      const int polls = B.tma_poll_limit > 0 ? B.tma_poll_limit : kTmaWaitPolls;
      if (tid == 0 && !B.tma_skip)
        tma_load_3d(tile, B.tmaps + j, bx * 32 - 8, by * R - H, 0, &bar,
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
    if constexpr (kStaged) {
      const float* plane0 = tile;
      const float* plane1 = tile + box_rows * kTileCols;
      const auto ref = tile_ref<H == 5 ? 4 : 1>(plane0, plane1, pair, parity, ty);
      sweep_pixel_staged<H>(J, pc, ref, inside, x, y, color, iter + J.iter_offset, wb);
    } else {
      int counts[2] = {0, 0};  // hypotheses, source windows sampled
      if (inside) {
        if constexpr (H > 0) {
          const float* plane0 = tile;
          const float* plane1 = tile + box_rows * kTileCols;
          const auto ref = tile_ref<4>(plane0, plane1, pair, parity, ty);
          const RefWindow rw = tile_window<H>(J, ref, x, y);
          sweep_pixel<H, kMode>(J, pc, ref, rw, x, y, color, iter + J.iter_offset, counts);
        } else {
          const GlobalRef<kCut> ref{J.pref, J.w, x, y};
          const RefWindow rw = ref_window(J, x, y, J.half_pixel);
          sweep_pixel<H, kMode>(J, pc, ref, rw, x, y, color, iter + J.iter_offset, counts);
        }
      }
      // all lanes again: the pixels' loops end at different times
      if (J.eval_counter) add_counts(J, counts, 2);
    }
    __syncthreads();
  }
  if constexpr (kStaged) {
    // a box copy whose wait ran out gets one more bounded chance to land
    // before the block's shared memory is released
    if (wb.dead && threadIdx.x == 0) mbar_wait(wb.bar, wb.phase ^ 1u, wb.polls);
  }
}

// Final maps of every job of the batch.
__global__ void __launch_bounds__(128) k_plane_output(const __grid_constant__ PlaneBatch B) {
  int j, x, y;
  if (!pixel_item(B, &j, &x, &y)) return;
  const Job& J = B.jobs[j];
  const int idx = y * J.w + x;
  const float4 h = J.hyp[idx];
  const float c = J.cost[idx];
  float d = __int_as_float(0x7fc00000);
  float cf = 0.f;
  uint8_t sp = 0;
  if (c < 1e29f && h.x > 0.f) {
    const float dd = 1.0f / h.x;
    if (dd >= (float)J.min_depth && dd <= (float)J.max_depth) {
      d = dd;
      cf = 1.0f - fminf(1.0f, fmaxf(0.0f, c));
      sp = J.support[idx];
      atomicAdd(J.out_filled, 1u);
    }
  }
  J.out_depth[idx] = d;
  J.out_support[idx] = sp;
  J.out_conf[idx] = cf;
  if (J.out_normal) {
    J.out_normal[3 * idx] = h.y;
    J.out_normal[3 * idx + 1] = h.z;
    J.out_normal[3 * idx + 2] = h.w;
  }
  if (J.out_cost) J.out_cost[idx] = c;
}

// Plane-mode refinement: golden-section search on the inverse depth along
// the pixel's own plane normal over +-1 px of disparity, the reference's
// refinement schedule applied to the plane cost.  One loop with a single
// evaluation: with one at each of the schedule's five places, the window code
// outgrew the instruction cache (a batch of four maps up to 960x720, 6-10
// sources, 11x11: 44.4 -> 14.3 ms; 9 maps of 640x480, 7x7: 16.2 -> 6.4 ms).
template <int H, int kMode>
__global__ void __launch_bounds__(128, 4) k_plane_refine(const __grid_constant__ PlaneBatch B) {
  extern __shared__ float2 smem[];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  int j, x, y;
  if (!pixel_item(B, &j, &x, &y)) return;
  const Job& J = B.jobs[j];
  if (J.refine_iters <= 0 || J.refine_mode != 1) return;
  PCache pc{smem, 128, tid};
  const int idx = y * J.w + x;
  const float4 h0 = J.hyp[idx];
  const float c0 = J.cost[idx];
  if (!(c0 < 1e29f)) return;
  float rx, ry;
  fill_pcache(J, pc, x, y, &rx, &ry);
  const RefWindow rw = ref_window(J, x, y, J.half_pixel);
  const GlobalRef<> ref{J.pref, J.w, x, y};
  float best_d = h0.x, best_c = c0;
  int best_s = J.support[idx];
  float lo = fmaxf(J.rho_min, best_d - J.inv_per_px);
  float hi = fminf(J.rho_max, best_d + J.inv_per_px);
  if (hi > lo) {
    const float inv_phi = 0.618033988749895f;
    float c1 = hi - inv_phi * (hi - lo), c2 = lo + inv_phi * (hi - lo);
    HypCost f1{kCostInf, 0}, f2{kCostInf, 0};
    const int last = J.refine_iters + 2;
#pragma unroll 1
    for (int t = 0; t <= last; ++t) {  // both first points, the iterations, the midpoint
      float v = c1;
      bool left = t == 0;
      if (t == 1) {
        v = c2;
      } else if (t == last) {
        v = 0.5f * (lo + hi);
      } else if (t > 1) {
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
      }
      const HypCost f = eval_plane_hyp<H, kMode>(J, pc, x, y, rx, ry, v, h0.y, h0.z, h0.w, rw, ref, nullptr);
      if (t == last) {
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
  J.hyp[idx] = make_float4(best_d, h0.y, h0.z, h0.w);
  J.cost[idx] = best_c;
  J.support[idx] = (uint8_t)min(best_s, 255);
}

// Plane-mode Gauss-Newton refinement (refine mode 2): Levenberg-Marquardt
// steps on (d, theta, phi) from the adjoint of the aggregated cost (exact
// bilinear reads, window recomputed per pass), each step accepted only when
// the search's own cost of the new plane is lower.
// The gradient and Gauss-Newton matrix of the aggregated cost for one
// refinement step: each view's moments (and from them the best_k selection)
// by the search's own window code with exact 2x2 reads -- an incremental
// homography walk -- then the adjoint's Jacobian pass over the selected
// views only.  False for an invalid hypothesis.
template <int H, int kMode, class Ref>
__device__ bool gn_gradient(const Job& J, const PCache& pc, int x, int y, float rx, float ry, const AdjHyp& h,
                            const RefWindow& rw, const Ref& ref, float g[3], float Hm[6]) {
  constexpr int kExact = kMode == kSrcBf16 ? kSrcBf16 : kSrcExact;
  for (int i = 0; i < 3; ++i) g[i] = 0.f;
  for (int i = 0; i < 6; ++i) Hm[i] = 0.f;
  PlaneHyp hp;
  if (!make_plane_hyp(J, rx, ry, 1.0f / h.d, h.n[0], h.n[1], h.n[2], &hp)) return false;
  const int ns = min(J.num_src, kMaxSources);
  ViewMom mom[kMaxSources];
  float vc[kMaxSources];
  int nvalid = 0;
  for (int s = 0; s < ns; ++s) {
    ff P[3];
    pc.get(s, P);
    float m[6];
    const ViewResult v = eval_view_plane<H, kExact>(J, J.src[s], x, y, P, hp, rw, ref, m);
    mom[s].valid = v.valid > 0;
    vc[s] = kCostInf;
    if (mom[s].valid) {
      mom[s].n = m[0];
      mom[s].mr = m[1];
      mom[s].ms = m[2];
      mom[s].srr = m[3];
      mom[s].sss = m[4];
      mom[s].srs = m[5];
      mom[s].ncc = v.ncc;
      vc[s] = 1.0f - v.ncc;
      ++nvalid;
    }
  }
  if (nvalid == 0) return false;
  const int k = (J.best_k <= 0 || J.best_k >= nvalid || J.best_k > kMaxBestK) ? nvalid : J.best_k;
  // the k lowest costs, ties to the lower source index
  uint32_t sel = 0;
  for (int t = 0; t < k; ++t) {
    int b = -1;
    for (int s = 0; s < ns; ++s)
      if (mom[s].valid && !((sel >> s) & 1u) && (b < 0 || vc[s] < vc[b])) b = s;
    sel |= 1u << b;
  }
  const float inv_k = 1.0f / (float)k;
  for (int s = 0; s < ns; ++s) {
    if (!((sel >> s) & 1u)) continue;
    float gs[3], Hs[6];
    const ViewGeo geo = view_geo(J, J.src[s], h);
    view_adjoint<kMode, false>(J, J.src[s], geo, h, mom[s], gs, Hs, nullptr, nullptr);
    for (int i = 0; i < 3; ++i) g[i] += gs[i] * inv_k;
    for (int i = 0; i < 6; ++i) Hm[i] += Hs[i] * inv_k;
  }
  return true;
}

template <int H, int kMode>
__global__ void __launch_bounds__(128, 5) k_plane_refine_gn(const __grid_constant__ PlaneBatch B) {
  extern __shared__ float2 smem[];
  const int tid = threadIdx.y * 32 + threadIdx.x;
  int j, x, y;
  if (!pixel_item(B, &j, &x, &y)) return;
  const Job& J = B.jobs[j];
  if (J.refine_iters <= 0 || J.refine_mode != 2) return;
  PCache pc{smem, 128, tid};
  const int idx = y * J.w + x;
  const float4 h0 = J.hyp[idx];
  float cur = J.cost[idx];
  if (!(cur < 1e29f) || !(h0.x > 0.f)) return;
  int sup = J.support[idx];
  float rx, ry;
  fill_pcache(J, pc, x, y, &rx, &ry);
  const RefWindow rw = ref_window(J, x, y, J.half_pixel);
  const GlobalRef<4> ref{J.pref, J.w, x, y};
  float d = 1.0f / h0.x;
  float theta = acosf(fminf(1.0f, fmaxf(-1.0f, h0.w))), phi = atan2f(h0.z, h0.y);
  float4 best = h0;
  float lambda = 1e-3f;
  for (int it = 0; it < J.refine_iters; ++it) {
    AdjHyp ah;
    if (!make_adj_hyp(J, x, y, d, theta, phi, &ah)) break;
    float g[3], Hm[6];
    if (!gn_gradient<H, kMode>(J, pc, x, y, rx, ry, ah, rw, ref, g, Hm)) break;
    bool accepted = false;
    for (int t = 0; t < 4 && !accepted; ++t) {
      float step[3];
      if (!solve_lm3(Hm, g, lambda, step)) {
        lambda *= 10.0f;
        continue;
      }
      const float nd = d + step[0], nt = theta + step[1], np = phi + step[2];
      float n[3], dt[3], dp[3];
      sph_normal(nt, np, n, dt, dp);
      const HypCost hc =
          eval_plane_hyp<H, kMode>(J, pc, x, y, rx, ry, 1.0f / nd, n[0], n[1], n[2], rw, ref, nullptr, nullptr,
                                   J.prune ? cur : kCostInf);
      if (nd > 0.f && hc.cost < cur) {
        d = nd;
        theta = nt;
        phi = np;
        cur = hc.cost;
        sup = hc.support;
        best = make_float4(1.0f / nd, n[0], n[1], n[2]);
        lambda *= 0.3f;
        accepted = true;
      } else {
        lambda *= 10.0f;
      }
    }
    if (!accepted) break;
  }
  J.hyp[idx] = best;
  J.cost[idx] = cur;
  J.support[idx] = (uint8_t)min(sup, 255);
}

// ---------------------------------------------------------------------------
// image preparation
// ---------------------------------------------------------------------------
__global__ void k_prep_ref(const uint8_t* __restrict__ img, int w, int h, float* ref, float* box) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const float v = (float)img[y * w + x] - 128.0f;
  ref[y * w + x] = v;
  if (box) {
    // the reference's window sample at (x + 0.5, y + 0.5): an exact 2x2
    // average; defined for x <= w-2, y <= h-2 (SampleBilinear's range)
    const int x1 = min(x + 1, w - 1), y1 = min(y + 1, h - 1);
    const float s = (float)img[y * w + x] + (float)img[y * w + x1] + (float)img[y1 * w + x] + (float)img[y1 * w + x1];
    box[y * w + x] = 0.25f * s - 128.0f;
  }
}

// Even / odd column planes of the (I - 128) reference image:
// out[p][y][i] = ref[y][2i + p] for i < half_w (0 past the right edge), rows
// of `pitch` floats (the padding is zero).
__global__ void k_deinterleave(const float* __restrict__ ref, int w, int h, int half_w, int pitch, float* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= pitch || y >= h) return;
  for (int p = 0; p < 2; ++p) {
    const int x = 2 * i + p;
    out[((size_t)p * h + y) * pitch + i] = (i < half_w && x < w) ? ref[(size_t)y * w + x] : 0.f;
  }
}

// One staged source texel of (I - 128) in the storage format (0 FP32, 1 FP16,
// 2 BF16 bits), rounded to nearest even.
// One source texel, v = I - 128, in the storage format (0 FP32, 1 FP16,
// 2 BF16 bits, 3 the 8-bit intensity I rounded to nearest and clamped).
__device__ __forceinline__ void store_texel(void* out, size_t i, float v, int storage) {
  if (storage == 1)
    ((__half*)out)[i] = __float2half_rn(v);
  else if (storage == 2)
    ((unsigned short*)out)[i] = __bfloat16_as_ushort(__float2bfloat16_rn(v));
  else if (storage == 3)
    ((uint8_t*)out)[i] = (uint8_t)__float2int_rn(fminf(255.0f, fmaxf(0.0f, v + 128.0f)));
  else
    ((float*)out)[i] = v;
}

__global__ void k_prep_src(const uint8_t* __restrict__ img, int w, int h, void* out, size_t pitch_elems,
                           int storage) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  store_texel(out, y * pitch_elems + x, (float)img[y * w + x] - 128.0f, storage);
}

__global__ void k_prep_ref_f32(const float* __restrict__ img, int w, int h, float* ref, float* box) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  ref[y * w + x] = img[y * w + x] - 128.0f;
  if (box) {
    const int x1 = min(x + 1, w - 1), y1 = min(y + 1, h - 1);
    const float s = (img[y * w + x] + img[y * w + x1]) + (img[y1 * w + x] + img[y1 * w + x1]);
    box[y * w + x] = 0.25f * s - 128.0f;
  }
}

__global__ void k_prep_src_f32in(const float* __restrict__ img, int w, int h, void* out, size_t pitch_elems,
                                 int storage) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  store_texel(out, y * pitch_elems + x, img[y * w + x] - 128.0f, storage);
}

// ComputeNcc (patchmatch_stereo.cpp:214-274) for a batch of windows, FP64 in
// the reference's operation order: a standalone API, not the hot path.
__device__ __forceinline__ bool sample_bilinear_d(const uint8_t* img, int w, int h, double u, double v, double* out) {
  if (u < 0.0 || v < 0.0 || u > (double)(w - 1) || v > (double)(h - 1)) return false;
  const int x0 = (int)floor(u), y0 = (int)floor(v);
  const int x1 = min(x0 + 1, w - 1), y1 = min(y0 + 1, h - 1);
  const double fx = __dsub_rn(u, (double)x0), fy = __dsub_rn(v, (double)y0);
  const double p00 = img[y0 * w + x0], p10 = img[y0 * w + x1], p01 = img[y1 * w + x0], p11 = img[y1 * w + x1];
  const double top = __dadd_rn(__dmul_rn(p00, __dsub_rn(1.0, fx)), __dmul_rn(p10, fx));
  const double bot = __dadd_rn(__dmul_rn(p01, __dsub_rn(1.0, fx)), __dmul_rn(p11, fx));
  *out = __dadd_rn(__dmul_rn(top, __dsub_rn(1.0, fy)), __dmul_rn(bot, fy));
  return true;
}

// One window's moments -> the result (the reference's tests and order).
__device__ __forceinline__ void store_ncc(int i, int patch_size, int valid, double sr, double ss, double srr,
                                          double sss, double srs, int* valid_out, double* ncc_out, int* weak_out,
                                          int* samples_out) {
  int ok = 0, weak = 0;
  double ncc = 0.0;
  if (valid >= patch_size * patch_size / 2) {
    const double nn = (double)valid;
    const double mr = __ddiv_rn(sr, nn), ms = __ddiv_rn(ss, nn);
    const double var_r = __dsub_rn(__ddiv_rn(srr, nn), __dmul_rn(mr, mr));
    const double var_s = __dsub_rn(__ddiv_rn(sss, nn), __dmul_rn(ms, ms));
    weak = var_r < 12.0;
    const double denom = __dsqrt_rn(__dmul_rn(var_r, var_s));
    if (!(denom < 1e-9)) {
      ncc = __ddiv_rn(__dsub_rn(__ddiv_rn(srs, nn), __dmul_rn(mr, ms)), denom);
      ncc = fmin(1.0, fmax(-1.0, ncc));
      ok = 1;
    }
  }
  valid_out[i] = ok;
  ncc_out[i] = ok ? ncc : 0.0;
  weak_out[i] = weak;
  samples_out[i] = ok ? valid : 0;
}

// Many windows: one thread each.
__global__ void k_ncc_windows(const uint8_t* __restrict__ ref, int ref_w, int ref_h, const uint8_t* __restrict__ src,
                              int src_w, int src_h, int patch_size, int n, const NccWindow* __restrict__ win,
                              int* valid_out, double* ncc_out, int* weak_out, int* samples_out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const NccWindow w = win[i];
  const int half = patch_size / 2;
  double sr = 0, ss = 0, srr = 0, sss = 0, srs = 0;
  int valid = 0;
  for (int dy = -half; dy <= half; ++dy)
    for (int dx = -half; dx <= half; ++dx) {
      double vr, vs;
      if (!sample_bilinear_d(ref, ref_w, ref_h, __dadd_rn(w.ref_u, (double)dx), __dadd_rn(w.ref_v, (double)dy), &vr))
        continue;
      if (!sample_bilinear_d(src, src_w, src_h, __dadd_rn(w.src_u, (double)dx), __dadd_rn(w.src_v, (double)dy), &vs))
        continue;
      sr = __dadd_rn(sr, vr);
      ss = __dadd_rn(ss, vs);
      srr = __dadd_rn(srr, __dmul_rn(vr, vr));
      sss = __dadd_rn(sss, __dmul_rn(vs, vs));
      srs = __dadd_rn(srs, __dmul_rn(vr, vs));
      ++valid;
    }
  store_ncc(i, patch_size, valid, sr, ss, srr, sss, srs, valid_out, ncc_out, weak_out, samples_out);
}

// Few windows: one warp each.  The reference's five running sums are serial
// FP64 chains, but what is summed is not: the lanes sample 128 positions at a
// time into shared memory (an invalid one adds zeros, which leave a sum that
// started at +0 unchanged), then lanes 0-4 each run one sum over them in order.
// 64 windows of 11 x 11: 21 us, where a thread for each took 253 us; bound by the
// chain of 121 dependent FP64 additions.
constexpr int kNccWarps = 4, kNccChunk = 128;
__global__ void __launch_bounds__(32 * kNccWarps) k_ncc_windows_warp(
    const uint8_t* __restrict__ ref, int ref_w, int ref_h, const uint8_t* __restrict__ src, int src_w, int src_h,
    int patch_size, int n, const NccWindow* __restrict__ win, int* valid_out, double* ncc_out, int* weak_out,
    int* samples_out) {
  __shared__ double term[kNccWarps][5][kNccChunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * kNccWarps + warp;
  if (i >= n) return;
  const NccWindow w = win[i];
  const int half = patch_size / 2, K = 2 * half + 1, total = K * K;
  double sum = 0.0;  // lanes 0-4: sr, ss, srr, sss, srs
  int valid = 0;
  for (int base = 0; base < total; base += kNccChunk) {
    const int m = min(kNccChunk, total - base);
#pragma unroll
    for (int j = 0; j < kNccChunk / 32; ++j) {
      const int t = base + j * 32 + lane;
      bool ok = t < total;
      double vr = 0.0, vs = 0.0;
      if (ok) {
        const int dy = t / K - half, dx = t % K - half;
        ok = sample_bilinear_d(ref, ref_w, ref_h, __dadd_rn(w.ref_u, (double)dx), __dadd_rn(w.ref_v, (double)dy), &vr) &&
             sample_bilinear_d(src, src_w, src_h, __dadd_rn(w.src_u, (double)dx), __dadd_rn(w.src_v, (double)dy), &vs);
      }
      if (!ok) vr = vs = 0.0;
      valid += ok;
      term[warp][0][j * 32 + lane] = vr;
      term[warp][1][j * 32 + lane] = vs;
      term[warp][2][j * 32 + lane] = __dmul_rn(vr, vr);
      term[warp][3][j * 32 + lane] = __dmul_rn(vs, vs);
      term[warp][4][j * 32 + lane] = __dmul_rn(vr, vs);
    }
    __syncwarp();
    if (lane < 5) {
#pragma unroll 8
      for (int e = 0; e < m; ++e) sum = __dadd_rn(sum, term[warp][lane][e]);
    }
    __syncwarp();
  }
  valid = (int)__reduce_add_sync(0xffffffffu, (unsigned int)valid);
  const double sr = __shfl_sync(0xffffffffu, sum, 0), ss = __shfl_sync(0xffffffffu, sum, 1),
               srr = __shfl_sync(0xffffffffu, sum, 2), sss = __shfl_sync(0xffffffffu, sum, 3),
               srs = __shfl_sync(0xffffffffu, sum, 4);
  if (lane == 0)
    store_ncc(i, patch_size, valid, sr, ss, srr, sss, srs, valid_out, ncc_out, weak_out, samples_out);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
cudaError_t launch_eval_hyps(const Job& J, int mode, int n, const int* px, const int* py, const double* inv,
                             const float* normals, float* cost, int* support, float* view_cost, cudaStream_t st) {
  const int threads = 128;
  const int blocks = (n + threads - 1) / threads;
  if (blocks == 0) return cudaSuccess;
  if (mode == 0) return launch_eval_compat_hyps(J, n, px, py, inv, cost, support, view_cost, st);
  const size_t sm = pcache_bytes(J.num_src, threads);
  return dispatch_plane(J.patch_half, J.src_mode, [&](auto h, auto k) {
    auto* fn = k_eval_hyps<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<blocks, threads, sm, st>>>(J, n, px, py, inv, normals, cost, support, view_cost);
    return cudaGetLastError();
  });
}

cudaError_t launch_plane_init(const PlaneBatch& B, int patch_half, int mode, int max_src, int* queues, int num_queues,
                              cudaStream_t st) {
  const int total = B.start[B.njobs];
  if (total <= 0) return cudaSuccess;
  const size_t sm = pcache_bytes(max_src, 128);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_init<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<total, dim3(32, 4), sm, st>>>(B, queues, num_queues);
    return cudaGetLastError();
  });
}

// The staged schedule's dynamic shared memory: the warps' boxes (after up to
// 128 bytes of alignment) and then the source-ray cache.
static size_t sweep_smem_bytes(int max_src, int rows, bool staged) {
  return pcache_bytes(max_src, 32 * rows) + (staged ? 128 + (size_t)rows * kStageBytes : 0);
}

// Calls f(kernel) for the sweep instance of (window, mode, schedule).
template <class F>
static cudaError_t dispatch_sweep(int patch_half, int mode, int staged, F&& f) {
  if (staged) {
    if (mode != kSrcExact) return cudaErrorInvalidValue;
    if (patch_half == 5) return f(k_plane_sweep<5, kSrcExact, true>);
    if (patch_half == 3) return f(k_plane_sweep<3, kSrcExact, true>);
    return cudaErrorInvalidValue;
  }
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    constexpr int H = decltype(h)::value, kMode = decltype(k)::value;
    // rows of 3, 5 and 9 samples waste fewer reads in groups of 3 than of 4
    // (640x480, 4 sources, exact reads, four half-sweeps: 3x3 2.31 -> 2.12 ms, 5x5
    // 3.98 -> 3.77, 9x9 9.2 -> 8.9; 15x15 21.8 -> 22.0)
    if constexpr (H == 0)
      if (patch_half == 1 || patch_half == 2 || patch_half == 4) return f(k_plane_sweep<0, kMode, false, 3>);
    return f(k_plane_sweep<H, kMode, false>);
  });
}

cudaError_t plane_sweep_occupancy(int patch_half, int mode, int max_src, int rows, int staged, int* blocks_per_sm) {
  const size_t sm = sweep_smem_bytes(max_src, rows, staged != 0);
  return dispatch_sweep(patch_half, mode, staged, [&](auto* fn) {
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, fn, 32 * rows, sm);
  });
}

cudaError_t launch_plane_sweep(const PlaneBatch& B, int total, int* queue, int patch_half, int mode, int max_src,
                               int rows, int staged, int grid, int color, int iter, cudaStream_t st) {
  if (total <= 0) return cudaSuccess;
  if (rows < 1 || rows > kMaxTileRows || grid < 1 || total > B.start[B.njobs]) return cudaErrorInvalidValue;
  const size_t sm = sweep_smem_bytes(max_src, rows, staged != 0);
  return dispatch_sweep(patch_half, mode, staged, [&](auto* fn) {
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<grid, dim3(32, rows), sm, st>>>(B, total, queue, color, iter);
    return cudaGetLastError();
  });
}

__global__ void k_pair_image(cudaTextureObject_t tex, int w, int h, float2* out, int pitch) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const float a = tex2D<float>(tex, (float)x + 0.5f, (float)y + 0.5f);
  const float b = x + 1 < w ? tex2D<float>(tex, (float)x + 1.5f, (float)y + 0.5f) : 0.0f;
  out[(size_t)y * pitch + x] = make_float2(a, b);
}

cudaError_t launch_pair_image(cudaTextureObject_t tex, int w, int h, float2* out, int pitch, cudaStream_t st) {
  if (w < 1 || h < 1 || pitch < w) return cudaErrorInvalidValue;
  const dim3 b(32, 8);
  k_pair_image<<<grid2d(w, h, b), b, 0, st>>>(tex, w, h, out, pitch);
  return cudaGetLastError();
}

cudaError_t launch_plane_refine(const PlaneBatch& B, int patch_half, int mode, int max_src, cudaStream_t st) {
  const int total = B.start[B.njobs];
  if (total <= 0) return cudaSuccess;
  const size_t sm = pcache_bytes(max_src, 128);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_refine<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<total, dim3(32, 4), sm, st>>>(B);
    return cudaGetLastError();
  });
}

cudaError_t launch_plane_refine_gn(const PlaneBatch& B, int patch_half, int mode, int max_src, cudaStream_t st) {
  const int total = B.start[B.njobs];
  if (total <= 0) return cudaSuccess;
  const size_t sm = pcache_bytes(max_src, 128);
  return dispatch_plane(patch_half, mode, [&](auto h, auto k) {
    auto* fn = k_plane_refine_gn<decltype(h)::value, decltype(k)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<total, dim3(32, 4), sm, st>>>(B);
    return cudaGetLastError();
  });
}

cudaError_t launch_plane_output(const PlaneBatch& B, cudaStream_t st) {
  const int total = B.start[B.njobs];
  if (total <= 0) return cudaSuccess;
  k_plane_output<<<total, dim3(32, 4), 0, st>>>(B);
  return cudaGetLastError();
}

cudaError_t launch_prep_ref(const uint8_t* img, int w, int h, float* ref, float* box, cudaStream_t st) {
  const dim3 b(32, 8);
  k_prep_ref<<<grid2d(w, h, b), b, 0, st>>>(img, w, h, ref, box);
  return cudaGetLastError();
}

static size_t texel_bytes(int storage) { return storage == 0 ? 4 : storage == 3 ? 1 : 2; }

cudaError_t launch_prep_src(const uint8_t* img, int w, int h, void* out, size_t pitch_bytes, int storage,
                            cudaStream_t st) {
  const dim3 b(32, 8);
  k_prep_src<<<grid2d(w, h, b), b, 0, st>>>(img, w, h, out, pitch_bytes / texel_bytes(storage), storage);
  return cudaGetLastError();
}

cudaError_t launch_prep_ref_f32(const float* img, int w, int h, float* ref, float* box, cudaStream_t st) {
  const dim3 b(32, 8);
  k_prep_ref_f32<<<grid2d(w, h, b), b, 0, st>>>(img, w, h, ref, box);
  return cudaGetLastError();
}

cudaError_t launch_prep_src_f32in(const float* img, int w, int h, void* out, size_t pitch_bytes, int storage,
                                  cudaStream_t st) {
  const dim3 b(32, 8);
  k_prep_src_f32in<<<grid2d(w, h, b), b, 0, st>>>(img, w, h, out, pitch_bytes / texel_bytes(storage), storage);
  return cudaGetLastError();
}

cudaError_t launch_ncc_windows(const uint8_t* ref, int ref_w, int ref_h, const uint8_t* src, int src_w, int src_h,
                               int patch_size, int n, const NccWindow* win, int* valid, double* ncc, int* weak,
                               int* samples, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  // A thread per window takes the same time until the windows fill the chip's
  // schedulers (2.1 us a sample and lane: 25 us for 3x3, 265 for 11x11, 2030 for
  // 31x31, up to 19,456 windows); a warp per window takes 0.17 us a sample and 7.5
  // us besides for every 1000 windows (76 us for 8000 of 3x3, 225 of 11x11, 1520 of
  // 31x31).  They cross at 2800, 9400 and 12,100 windows; the line is a little below.
  const long long area = (long long)patch_size * patch_size;
  if (n * (area + 44) <= 11000 * area)
    k_ncc_windows_warp<<<(n + kNccWarps - 1) / kNccWarps, 32 * kNccWarps, 0, st>>>(
        ref, ref_w, ref_h, src, src_w, src_h, patch_size, n, win, valid, ncc, weak, samples);
  else
    k_ncc_windows<<<(n + 127) / 128, 128, 0, st>>>(ref, ref_w, ref_h, src, src_w, src_h, patch_size, n, win, valid,
                                                   ncc, weak, samples);
  return cudaGetLastError();
}

cudaError_t launch_deinterleave(const float* ref, int w, int h, int half_w, int pitch, float* out, cudaStream_t st) {
  const dim3 b(32, 8);
  k_deinterleave<<<grid2d(pitch, h, b), b, 0, st>>>(ref, w, h, half_w, pitch, out);
  return cudaGetLastError();
}


}  // namespace rmvs
