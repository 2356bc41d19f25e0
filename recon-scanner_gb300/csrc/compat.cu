// compat.cu -- compat mode (drop-in parity): the reference PatchMatchStereo's
// fronto-parallel Jacobi sweeps and RefineSubpixel, one thread per pixel; the
// reference's row-block xorshift draws are generated on the host in its scan
// order.  A warp's lanes go through candidates, steps and views together, those
// without a pixel or a candidate too: the window code votes (eval_view_compat).
#include "compat.cuh"

namespace rmvs {

// ---------------------------------------------------------------------------
// compat mode (the reference algorithm)
// ---------------------------------------------------------------------------
// Given hypotheses (the parity instrument), by the general window for every
// size.
__global__ void __launch_bounds__(128, 4) k_eval_compat_hyps(Job J, int n, const int* __restrict__ px,
                                                             const int* __restrict__ py, const double* __restrict__ inv,
                                                             float* out_cost, int* out_support, float* out_view_cost) {
  extern __shared__ float2 smem[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  PCache pc{smem, (int)blockDim.x, (int)threadIdx.x};
  const bool have = i < n;
  const int x = have ? px[i] : 0, y = have ? py[i] : 0;
  RefWindow rw{0.0f, 0.0f, false};
  if (have) {
    float rx, ry;
    fill_pcache(J, pc, x, y, &rx, &ry);
    rw = ref_window(J, x, y, true);
  }
  const HypCost r = eval_compat_hyp<0>(J, pc, x, y, have ? inv[i] : 0.0, have, rw, CompatRef<0>{},
                                       have && out_view_cost ? out_view_cost + (size_t)i * J.num_src : nullptr);
  if (!have) return;
  out_cost[i] = r.cost;
  out_support[i] = r.support;
}

template <int H>
__global__ void __launch_bounds__(128, 4) k_compat_init(Job J, float* cost) {
  extern __shared__ float2 smem[];
  __shared__ CompatTile<H> tile;
  load_compat_tile(J, tile);
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  PCache pc{smem, (int)(blockDim.x * blockDim.y), tid};
  const CompatRef<H> ref{&tile, (int)threadIdx.x, (int)threadIdx.y};
  const bool inside = x < J.w && y < J.h;
  const int idx = inside ? y * J.w + x : 0;
  RefWindow rw{0.0f, 0.0f, false};
  if (inside) {
    float rx, ry;
    fill_pcache(J, pc, x, y, &rx, &ry);
    rw = ref_window(J, x, y, true);
  }
  const HypCost c = eval_compat_hyp<H>(J, pc, x, y, inside ? J.inv[idx] : 0.0, inside, rw, ref, nullptr);
  if (!inside) return;
  cost[idx] = c.cost;
  J.isupport[idx] = c.support;
}

// One direction sweep (patchmatch_stereo.cpp:642-723) for every pixel at
// once: candidates come from the snapshot (inv_in, cost_in); the pixel's own
// draws -- random_search_count signed draws, the restart flag and the
// restart draw -- were generated on the host in the reference's scan order.
// One loop over the candidates (4 neighbours, the signed draws, the restart),
// so that the hypothesis evaluation is compiled once; a candidate is weighed
// against the pixel's current cost (eval_compat_hyp's `beat`).  These kernels are
// capped at 128 registers, 4 blocks an SM: uncapped, 11x11 and 17x17 at 640x480
// with 3 sources take the same or 13 % longer in the sweeps and 7 % in the
// refinement (16 warps hide more than the spills cost); 5 blocks, 96 registers,
// 10 to 30 % longer.
template <int H>
__global__ void __launch_bounds__(128, 4) k_compat_sweep(
    Job J, const double* __restrict__ inv_in, const float* __restrict__ cost_in, const int32_t* __restrict__ sup_in,
    double* inv_out, float* cost_out, int32_t* sup_out, const uint32_t* __restrict__ draws,
    const uint8_t* __restrict__ fire, int draw_stride, int search_count, double radius_ratio, int propagate) {
  extern __shared__ float2 smem[];
  __shared__ CompatTile<H> tile;
  load_compat_tile(J, tile);
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  PCache pc{smem, (int)(blockDim.x * blockDim.y), tid};
  const CompatRef<H> ref{&tile, (int)threadIdx.x, (int)threadIdx.y};
  const bool inside = x < J.w && y < J.h;
  const int idx = inside ? y * J.w + x : 0;
  RefWindow rw{0.0f, 0.0f, false};
  double out_inv = 0.0;
  float out_cost = kCostInf;
  int out_sup = 0;
  if (inside) {
    float rx, ry;
    fill_pcache(J, pc, x, y, &rx, &ry);
    rw = ref_window(J, x, y, true);
    out_inv = inv_in[idx];
    out_cost = cost_in[idx];
    out_sup = sup_in[idx];
  }
  const uint32_t* d = draws + (size_t)idx * draw_stride;
  double radius = 0.0;
#pragma unroll 1
  for (int k = propagate ? 0 : 4; k <= 4 + search_count; ++k) {
    double cand = 0.0;
    bool have = inside;
    if (k < 4) {
      const int nx_ = x + (k == 0 ? -1 : k == 1 ? 1 : 0), ny_ = y + (k == 2 ? -1 : k == 3 ? 1 : 0);
      have = have && nx_ >= 0 && ny_ >= 0 && nx_ < J.w && ny_ < J.h;
      const int n = have ? ny_ * J.w + nx_ : 0;
      have = have && !(cost_in[n] >= 1e29f);
      if (have) cand = inv_in[n];
    } else if (k < 4 + search_count) {
      // the search radius comes from the inverse depth after propagation
      if (k == 4) radius = out_inv * radius_ratio;
      const double sgn = ((double)d[k - 4] / 4294967296.0) * 2.0 - 1.0;
      cand = out_inv + sgn * radius;
      radius *= 0.5;
      have = have && !(cand < J.dinv_min || cand > J.dinv_max);
    } else {
      have = have && fire[idx];
      if (have) cand = J.dinv_min + ((double)d[search_count] / 4294967296.0) * (J.dinv_max - J.dinv_min);
    }
    const HypCost c = eval_compat_hyp<H>(J, pc, x, y, cand, have, rw, ref, nullptr, out_cost);
    if (have && c.cost < out_cost) {
      out_cost = c.cost;
      out_inv = cand;
      out_sup = c.support;
    }
  }
  if (!inside) return;
  inv_out[idx] = out_inv;
  cost_out[idx] = out_cost;
  sup_out[idx] = out_sup;
}

// patchmatch_stereo.cpp:744-763
__global__ void k_compat_output(Job J, const double* __restrict__ inv, const float* __restrict__ cost,
                                const int32_t* __restrict__ sup, float* depth, uint8_t* support, float* conf,
                                unsigned int* filled) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= J.w || y >= J.h) return;
  const int idx = y * J.w + x;
  float d = __int_as_float(0x7fc00000);
  float cf = 0.f;
  uint8_t sp = 0;
  if (cost[idx] < 1e29f) {
    const double iv = inv[idx];
    const double dd = iv <= 1e-9 ? 1e9 : 1.0 / iv;
    if (!(dd < J.min_depth || dd > J.max_depth)) {
      d = (float)dd;
      sp = (uint8_t)min(sup[idx], 255);
      const double pc = fmin(1.0, fmax(0.0, (double)cost[idx]));
      cf = (float)(1.0 - pc);
      atomicAdd(filled, 1u);
    }
  }
  depth[idx] = d;
  support[idx] = sp;
  conf[idx] = cf;
}

// RefineSubpixel (patchmatch_stereo.cpp:770-979), one thread per pixel.
// Inverse-depth arithmetic in FP64 as in the reference; costs FP32.
__device__ __forceinline__ bool solve3(const double A[3][3], const double b[3], double x[3]) {
  double m[3][4];
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j) m[i][j] = A[i][j];
    m[i][3] = b[i];
  }
  for (int col = 0; col < 3; ++col) {
    int pivot = col;
    for (int r = col + 1; r < 3; ++r)
      if (fabs(m[r][col]) > fabs(m[pivot][col])) pivot = r;
    if (fabs(m[pivot][col]) < 1e-18) return false;
    if (pivot != col)
      for (int j = 0; j < 4; ++j) {
        const double t = m[col][j];
        m[col][j] = m[pivot][j];
        m[pivot][j] = t;
      }
    for (int r = 0; r < 3; ++r) {
      if (r == col) continue;
      const double f = m[r][col] / m[col][col];
      for (int j = col; j < 4; ++j) m[r][j] -= f * m[col][j];
    }
  }
  for (int i = 0; i < 3; ++i) {
    if (fabs(m[i][i]) < 1e-18) return false;
    x[i] = m[i][3] / m[i][i];
  }
  return true;
}

// The steps of one pixel -- the fit points, the centre, the parabola's vertex,
// the golden section's first two points, its iterations, its midpoint -- run as
// one loop with a single evaluation, so that the window code is compiled once
// and a warp's lanes evaluate the same step together.
template <int H>
__global__ void __launch_bounds__(128, 4) k_compat_refine(Job J, float* depth, float* conf, double inv_per_px,
                                                       int fit_points_cfg, int subpixel_iterations,
                                                       unsigned int* refined, double* out_best_inv,
                                                       float* out_best_cost) {
  extern __shared__ float2 smem[];
  __shared__ CompatTile<H> tile;
  load_compat_tile(J, tile);
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int y = blockIdx.y * blockDim.y + threadIdx.y;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
  PCache pc{smem, (int)(blockDim.x * blockDim.y), tid};
  const CompatRef<H> ref{&tile, (int)threadIdx.x, (int)threadIdx.y};
  const bool inside = x < J.w && y < J.h;
  const int idx = inside ? y * J.w + x : 0;
  const float d0 = inside ? depth[idx] : 0.0f;
  if (out_best_inv && inside) {
    out_best_inv[idx] = __longlong_as_double(0x7ff8000000000000ll);
    out_best_cost[idx] = kCostInf;
  }
  const double inv0 = (double)d0 < 1e-9 ? 1e9 : 1.0 / (double)d0;
  const bool have = inside && isfinite(d0) && !(inv0 < J.dinv_min || inv0 > J.dinv_max);
  RefWindow rw{0.0f, 0.0f, false};
  if (have) {
    float rx, ry;
    fill_pcache(J, pc, x, y, &rx, &ry);
    rw = ref_window(J, x, y, true);
  }
  const int fit_points = fit_points_cfg > 3 ? fit_points_cfg : 3;
  const int half_fit = fit_points / 2;
  const double fit_step = inv_per_px * 0.5;
  double s0 = 0, s1 = 0, s2 = 0, s3 = 0, s4 = 0, t0 = 0, t1 = 0, t2 = 0;
  bool fit_ok = fit_points <= 64;
  const int fits = fit_ok ? fit_points : 0;
  bool have_centre = false;  // the middle fit point is the centre itself
  double best_d = inv0;
  float best_c = kCostInf;
  const double inv_phi = 0.6180339887498949;
  double lo = 0, hi = 0, c1 = 0, c2 = 0, v = 0;
  float f1 = 0, f2 = 0;
  bool section = false, left = false;
  const int first = fits + 2;  // the golden section's first step
  const int last = first + 2 + (subpixel_iterations > 0 ? subpixel_iterations : 0);
#pragma unroll 1
  for (int t = 0; t <= last; ++t) {
    bool want;
    if (t < fits) {
      v = inv0 + (t - half_fit) * fit_step;
      if (fit_ok && (v < J.dinv_min || v > J.dinv_max)) fit_ok = false;
      want = fit_ok;
    } else if (t == fits) {
      v = inv0;
      want = !have_centre;
    } else if (t == fits + 1) {
      want = false;
      if (fit_ok) {
        const double A[3][3] = {{s4, s3, s2}, {s3, s2, s1}, {s2, s1, s0}};
        const double b[3] = {t2, t1, t0};
        double sol[3];
        if (solve3(A, b, sol) && fabs(sol[0]) > 1e-12) {
          const double vertex = -sol[1] / (2.0 * sol[0]);
          // the vertex is in sample-index units and is added unscaled, as in
          // the reference (patchmatch_stereo.cpp:896-899)
          if (vertex >= -(double)half_fit && vertex <= (double)half_fit) {
            v = inv0 + vertex;
            want = true;
          }
        }
      }
    } else {
      if (t == first) {
        lo = best_d - inv_per_px * 1.0;
        hi = best_d + inv_per_px * 1.0;
        if (lo < J.dinv_min) lo = J.dinv_min;
        if (hi > J.dinv_max) hi = J.dinv_max;
        section = hi > lo;
        c1 = hi - inv_phi * (hi - lo);
        c2 = lo + inv_phi * (hi - lo);
        v = c1;
      } else if (t == first + 1) {
        v = c2;
      } else if (t < last) {
        left = f1 < f2;
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
        v = 0.5 * (lo + hi);
      }
      want = section;
    }
    want = want && have;
    const float fc = eval_compat_hyp<H>(J, pc, x, y, v, want, rw, ref, nullptr).cost;
    if (!want) continue;
    if (t < fits) {
      const double c = (double)fc;
      if (c >= 1e29) fit_ok = false;
      if (t == half_fit) {
        have_centre = true;
        best_c = fc;
      }
      const double xx = (double)(t - half_fit);
      s0 += 1.0;
      s1 += xx;
      s2 += xx * xx;
      s3 += xx * xx * xx;
      s4 += xx * xx * xx * xx;
      t0 += c;
      t1 += xx * c;
      t2 += xx * xx * c;
    } else if (t == fits) {
      best_c = fc;
    } else if (t == fits + 1) {
      if (fc < best_c) {
        best_c = fc;
        best_d = v;
      }
    } else if (t == first) {
      f1 = fc;
    } else if (t == first + 1) {
      f2 = fc;
    } else if (t < last) {
      if (left)
        f1 = fc;
      else
        f2 = fc;
    } else {
      if (fc < best_c) {
        best_c = fc;
        best_d = v;
      }
      if (f1 < best_c) {
        best_c = f1;
        best_d = c1;
      }
      if (f2 < best_c) {
        best_c = f2;
        best_d = c2;
      }
    }
  }
  if (!have) return;
  if (out_best_inv) {
    out_best_inv[idx] = best_d;
    out_best_cost[idx] = best_c;
  }
  if (best_d < J.dinv_min || best_d > J.dinv_max) return;
  const double fd = best_d <= 1e-9 ? 1e9 : 1.0 / best_d;
  if (fd < J.min_depth || fd > J.max_depth) return;
  depth[idx] = (float)fd;
  const double pcost = fmin(1.0, fmax(0.0, (double)best_c));
  conf[idx] = (float)(1.0 - pcost);
  atomicAdd(refined, 1u);
}

// Calls f(integral_constant<H>) for a window of 2 patch_half + 1: compiled whole
// from 3x3 to 17x17, the general loop (0) for any other.  The line lies where
// the whole form has been measured: it beats the general loop at every size
// below (3 sources, 640x480, four sweeps and the refinement: 3x3 1.11 and 0.44
// ms against 1.52 and 0.52; 17x17 6.3 and 1.8 ms against 21.7 and 6.1 of the
// general loop at its best), and each size is three more kernels to build.
template <class F>
static cudaError_t dispatch_compat(int patch_half, F&& f) {
  using std::integral_constant;
  switch (patch_half) {
    case 1: return f(integral_constant<int, 1>{});
    case 2: return f(integral_constant<int, 2>{});
    case 3: return f(integral_constant<int, 3>{});
    case 4: return f(integral_constant<int, 4>{});
    case 5: return f(integral_constant<int, 5>{});
    case 6: return f(integral_constant<int, 6>{});
    case 7: return f(integral_constant<int, 7>{});
    case 8: return f(integral_constant<int, 8>{});
    default: return f(integral_constant<int, 0>{});
  }
}

cudaError_t launch_eval_compat_hyps(const Job& J, int n, const int* px, const int* py, const double* inv, float* cost,
                                    int* support, float* view_cost, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const size_t sm = pcache_bytes(J.num_src, 128);
  cudaError_t e = allow_smem(k_eval_compat_hyps, sm);
  if (e != cudaSuccess) return e;
  k_eval_compat_hyps<<<(n + 127) / 128, 128, sm, st>>>(J, n, px, py, inv, cost, support, view_cost);
  return cudaGetLastError();
}

cudaError_t launch_compat_init(const Job& J, float* cost, cudaStream_t st) {
  const dim3 b(32, kCompatRows);
  const size_t sm = pcache_bytes(J.num_src, 128);
  return dispatch_compat(J.patch_half, [&](auto h) {
    auto* fn = k_compat_init<decltype(h)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<grid2d(J.w, J.h, b), b, sm, st>>>(J, cost);
    return cudaGetLastError();
  });
}

cudaError_t launch_compat_sweep(const Job& J, const double* inv_in, const float* cost_in, const int32_t* sup_in,
                                double* inv_out, float* cost_out, int32_t* sup_out, const uint32_t* draws,
                                const uint8_t* fire, int draw_stride, int search_count, double radius_ratio,
                                int propagate, cudaStream_t st) {
  const dim3 b(32, kCompatRows);
  const size_t sm = pcache_bytes(J.num_src, 128);
  return dispatch_compat(J.patch_half, [&](auto h) {
    auto* fn = k_compat_sweep<decltype(h)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<grid2d(J.w, J.h, b), b, sm, st>>>(J, inv_in, cost_in, sup_in, inv_out, cost_out, sup_out, draws, fire,
                                           draw_stride, search_count, radius_ratio, propagate);
    return cudaGetLastError();
  });
}

cudaError_t launch_compat_output(const Job& J, const double* inv, const float* cost, const int32_t* sup, float* depth,
                                 uint8_t* support, float* conf, unsigned int* filled, cudaStream_t st) {
  const dim3 b(32, 8);
  k_compat_output<<<grid2d(J.w, J.h, b), b, 0, st>>>(J, inv, cost, sup, depth, support, conf, filled);
  return cudaGetLastError();
}

cudaError_t launch_compat_refine(const Job& J, float* depth, float* conf, double inv_per_px, int fit_points,
                                 int iters, unsigned int* refined, double* best_inv, float* best_cost,
                                 cudaStream_t st) {
  const dim3 b(32, kCompatRows);
  const size_t sm = pcache_bytes(J.num_src, 128);
  return dispatch_compat(J.patch_half, [&](auto h) {
    auto* fn = k_compat_refine<decltype(h)::value>;
    cudaError_t e = allow_smem(fn, sm);
    if (e != cudaSuccess) return e;
    fn<<<grid2d(J.w, J.h, b), b, sm, st>>>(J, depth, conf, inv_per_px, fit_points, iters, refined, best_inv,
                                           best_cost);
    return cudaGetLastError();
  });
}

}  // namespace rmvs
