// tsdf.cu -- TSDF fusion of depth frames into a device-resident voxel grid.
//
// The reference's TsdfVolume (core/src/rgbd/tsdf_fusion.cpp with the shared
// kernel core/src/rgbd/tsdf_internal.h) walks each valid pixel's viewing ray
// across the truncation band and folds every voxel it meets into a running
// weighted mean, pixel after pixel in raster order.  A voxel can be met by
// many pixels of one frame, and floating-point running means depend on their
// order, so the GPU keeps it: every (pixel, step) pair is one update record
// whose place in the reference's order is known from its index; the records of
// a voxel are chained to it, and a thread per touched voxel (a warp, for a long
// chain) brings its chain back into record order and folds it in sequence.  The grid -- and the surface
// points extracted from it -- are bit-identical to the reference's.  FP64 and
// FP32 arithmetic that reaches the grid is written with explicit
// round-to-nearest operations in the reference's evaluation order (no
// contractions); a cheaper form stands in for it only where a test shows that
// both round to the same value.
//
// Layout in HBM: tsdf and weight as FP32 arrays over the dense grid, index
// (iz * ny + iy) * nx + ix, as in the reference (8 bytes per voxel; the
// reference also keeps 12 bytes of colour it never writes).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <new>
#include <string>

#include "kernels.h"
#include "pool.h"
#include "recon_mvs_gb300.h"

namespace rmvs {

extern thread_local std::string g_last_error;

namespace {

struct TsdfFrame {
  int w, h;
  int nx, ny, nz;
  int steps;
  float voxel, trunc, w_new;
  double fx, fy, cx, cy, min_depth, max_depth;
  int min_conf;
  double origin[3];
  double R_wc[9], t_wc[3], R_cw[9], t_cw[3];
  double inv_trunc;            // 1 / truncation, FP64
  float Rf[9], tf[3];          // R_wc, t_wc in FP32 (the projection's estimate)
  float r_scale;               // the largest |R_wc| entry, at least 1
  int rotation;                // R_wc is orthonormal to 4e-16: |R p| is |p| to 1e-15
  const double* dir_x;         // (u - cx) / fx per column
  const double* dir_y;         // (v - cy) / fy per row
  const double* depth_of[3];   // R_wc[2][axis] * the voxel centre's coordinate, per axis
};

constexpr unsigned int kNoRecord = 0xffffffffu;

// A voxel centre's coordinate on one axis (VoxelToWorld in FP32).
__device__ __forceinline__ float voxel_centre(float origin, int i, float voxel) {
  return __fadd_rn(origin, __fmul_rn(__fadd_rn((float)i, 0.5f), voxel));
}

__device__ __forceinline__ void mat3_vec_rn(const double* m, const double* v, double* out) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // the reference's sum starts at +0: 0 + x is x (a zero's sign is not used)
    double s = __dmul_rn(m[i * 3], v[0]);
#pragma unroll
    for (int j = 1; j < 3; ++j) s = __dadd_rn(s, __dmul_rn(m[i * 3 + j], v[j]));
    out[i] = s;
  }
}

__device__ __forceinline__ void normalized_rn(const double* v, double* out) {
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) s = __dadd_rn(s, __dmul_rn(v[i], v[i]));
  const double n = __dsqrt_rn(s);
  if (n < 1e-15) {
    out[0] = out[1] = out[2] = 0.0;
    return;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) out[i] = __ddiv_rn(v[i], n);
}

__device__ __forceinline__ int floor_scaled(float a, float b) { return (int)floorf(__fdiv_rn(a, b)); }

// floor(fl(a / b)) of FP32 values with inv_b = fl(1 / b): the product is within a
// few ulp of the quotient, so the division is needed only beside an integer.
__device__ __forceinline__ int floor_quotient(float a, float b, float inv_b) {
  const float q = a * inv_b;
  const float f = floorf(q), r = q - f;
  if (r > 1e-3f && r < 1.0f - 1e-3f && fabsf(q) < 1024.0f) return (int)f;
  return floor_scaled(a, b);
}

// fl32(fl64(diff / trunc)) from diff * (1 / trunc): within 2 ulp (FP64) of the
// quotient, so both round to the same float unless the 29 bits that the
// rounding drops are within 4 of a half (or the float is subnormal).
__device__ __forceinline__ float truncated_sdf(double diff, double trunc, double inv_trunc) {
  const double q = __dmul_rn(diff, inv_trunc);
  const int low = (int)((unsigned int)__double2loint(q) & 0x1fffffffu) - 0x10000000;
  if ((low >= -4 && low <= 4) || (__double2hiint(q) & 0x7fffffff) < 0x38500000)
    return __double2float_rn(__ddiv_rn(diff, trunc));
  return __double2float_rn(q);
}

// The FP32 direction of the walk, fl32(normalize(R_cw normalize(p))): from
// R_cw p and 1 / |p| (an FP32 seed and two Newton steps) in 18 FP64 operations
// instead of the 115 of two square roots and six divisions.  The result is
// within 2e-15 of the reference's FP64 vector, so both round to the same float
// unless a component is small or its dropped bits are beside a half: false then.
__device__ __forceinline__ bool walk_direction(const double p[3], const double rp[3], float out[3]) {
  const double pp = fma(p[0], p[0], fma(p[1], p[1], p[2] * p[2]));
  const float ppf = (float)pp;
  double y = (double)rsqrtf(ppf);
#pragma unroll
  for (int i = 0; i < 2; ++i) y = fma(0.5 * y, fma(-pp * y, y, 1.0), y);
  bool sure = ppf > 1e-20f && ppf < 1e20f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double n = rp[i] * y;
    const int low = (int)((unsigned int)__double2loint(n) & 0x1fffffffu) - 0x10000000;
    out[i] = __double2float_rn(n);
    // 2e-15 is below 2^14 ulp of a component of at least 1e-3
    sure = sure && fabsf(out[i]) >= 1e-3f && fabsf(out[i]) <= 1.5f && (low < -16384 || low > 16384);
  }
  return sure;
}

// The per-frame tables: viewing-ray slopes per column and row, and per axis
// the voxel centres' terms of the camera depth, each in the reference's own
// FP64 operations -- per pixel and step they would be repeated a hundred times.
__global__ void k_tsdf_tables(TsdfFrame F, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int k = i;
  if (k < F.w) {
    out[i] = __ddiv_rn(__dsub_rn((double)k, F.cx), F.fx);
    return;
  }
  k -= F.w;
  if (k < F.h) {
    out[i] = __ddiv_rn(__dsub_rn((double)k, F.cy), F.fy);
    return;
  }
  k -= F.h;
  const int n[3] = {F.nx, F.ny, F.nz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (k < n[a]) {
      out[i] = __dmul_rn(F.R_wc[6 + a], (double)voxel_centre(__double2float_rn(F.origin[a]), k, F.voxel));
      return;
    }
    k -= n[a];
  }
}

// One thread per pixel: the updates of its ray walk.  Record r = pixel * steps +
// step (its place in the reference's order) holds {the voxel's previous record,
// sdf} and heads the voxel's chain from then on; `first[step * pixels + pixel]`
// is the voxel when the record is the first of its chain, else -1.  What bounded
// this kernel is FP64 issue (2 operations a cycle and SM): about 65 a step for
// the transform, the projection's two divisions and the sdf's, and 150 a pixel.
// Only the depth and the sdf reach the grid; the depth is three additions of
// tabled products, the sdf a product (truncated_sdf), and the projection, which
// only has to be inside the frame, is decided in FP32 unless it falls within its
// error of an edge: 6 FP64 operations a step, about 50 a pixel.  640x480, 19
// steps: 0.69 -> 0.18 ms a frame, FP64 still the busiest pipe.
__global__ void __launch_bounds__(256) k_tsdf_walk(TsdfFrame F, const uint16_t* __restrict__ depth,
                                                   const uint8_t* __restrict__ conf, unsigned int* head, uint2* rec,
                                                   int* first, unsigned int* integrated) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  const int v = blockIdx.y * blockDim.y + threadIdx.y;
  const bool in_frame = u < F.w && v < F.h;
  const unsigned int pix = in_frame ? (unsigned int)v * F.w + u : 0u;
  const unsigned int npix = (unsigned int)F.w * F.h;
  const uint16_t d_raw = in_frame ? depth[pix] : 0;
  bool ok = d_raw != 0;
  if (ok && conf && (int)conf[pix] < F.min_conf) ok = false;
  const double d = __dmul_rn((double)d_raw, 1e-3);
  if (d < F.min_depth || d > F.max_depth) ok = false;
  const int n_ok = __syncthreads_count(ok);
  if (threadIdx.x == 0 && threadIdx.y == 0 && n_ok) atomicAdd(integrated, (unsigned int)n_ok);
  if (!in_frame) return;
  if (!ok) {
    for (int s = 0; s <= 2 * F.steps; ++s) first[(size_t)s * npix + pix] = -1;
    return;
  }
  const double p_cam[3] = {__dmul_rn(F.dir_x[u], d), __dmul_rn(F.dir_y[v], d), d};
  double rp[3], pw[3];
  mat3_vec_rn(F.R_cw, p_cam, rp);
#pragma unroll
  for (int i = 0; i < 3; ++i) pw[i] = __dadd_rn(rp[i], F.t_cw[i]);
  float dir[3];
  if (!F.rotation || !walk_direction(p_cam, rp, dir)) {
    double ray[3], rw[3], nw[3];
    normalized_rn(p_cam, ray);
    mat3_vec_rn(F.R_cw, ray, rw);
    normalized_rn(rw, nw);
#pragma unroll
    for (int i = 0; i < 3; ++i) dir[i] = __double2float_rn(nw[i]);
  }
  const int cxv = floor_scaled(__double2float_rn(__dsub_rn(pw[0], F.origin[0])), F.voxel);
  const int cyv = floor_scaled(__double2float_rn(__dsub_rn(pw[1], F.origin[1])), F.voxel);
  const int czv = floor_scaled(__double2float_rn(__dsub_rn(pw[2], F.origin[2])), F.voxel);
  const float nxw = dir[0], nyw = dir[1], nzw = dir[2];
  const float ox = __double2float_rn(F.origin[0]), oy = __double2float_rn(F.origin[1]),
              oz = __double2float_rn(F.origin[2]);
  const double trunc = (double)F.trunc;
  const float inv_voxel = 1.0f / F.voxel;
  const unsigned int nst = 2u * F.steps + 1u;
  const float fxf = (float)F.fx, fyf = (float)F.fy, cxf = (float)F.cx, cyf = (float)F.cy;
#pragma unroll 1
  for (int s = -F.steps; s <= F.steps; ++s) {
    const unsigned int r = pix * nst + (unsigned int)(s + F.steps);
    int voxel_of_first = -1;
    const float dist = __fmul_rn((float)s, F.voxel);
    const int ix = cxv + floor_quotient(__fmul_rn(dist, nxw), F.voxel, inv_voxel);
    const int iy = cyv + floor_quotient(__fmul_rn(dist, nyw), F.voxel, inv_voxel);
    const int iz = czv + floor_quotient(__fmul_rn(dist, nzw), F.voxel, inv_voxel);
    if (ix >= 0 && iy >= 0 && iz >= 0 && ix < F.nx && iy < F.ny && iz < F.nz) {
      const double zc = __dadd_rn(__dadd_rn(__dadd_rn(F.depth_of[0][ix], F.depth_of[1][iy]), F.depth_of[2][iz]),
                                  F.t_wc[2]);
      const double diff = __dsub_rn(d, zc);
      // FP64 comparisons of non-negative values as integers (a negative or NaN
      // depth fails the first, a NaN difference the second)
      if (__double_as_longlong(zc) > __double_as_longlong(1e-6) &&
          (__double_as_longlong(diff) & 0x7fffffffffffffffll) <= __double_as_longlong(trunc)) {
        // the projection in FP32: each coordinate is within `e` of the exact one
        const float vx = voxel_centre(ox, ix, F.voxel), vy = voxel_centre(oy, iy, F.voxel),
                    vz = voxel_centre(oz, iz, F.voxel);
        const float X = fmaf(F.Rf[0], vx, fmaf(F.Rf[1], vy, fmaf(F.Rf[2], vz, F.tf[0])));
        const float Y = fmaf(F.Rf[3], vx, fmaf(F.Rf[4], vy, fmaf(F.Rf[5], vz, F.tf[1])));
        const float Z = fmaf(F.Rf[6], vx, fmaf(F.Rf[7], vy, fmaf(F.Rf[8], vz, F.tf[2])));
        const float iZ = rcp_approx(Z);
        const float size = F.r_scale * (fabsf(vx) + fabsf(vy) + fabsf(vz)) + fabsf(F.tf[0]) + fabsf(F.tf[1]) +
                           fabsf(F.tf[2]);
        const float qx = X * iZ, qy = Y * iZ;
        const float ux = fmaf(fxf, qx, cxf), uy = fmaf(fyf, qy, cyf);
        // at most 8 roundings of 2^-24, on terms of at most `size`
        const float e = 0.01f +
                        2e-6f * (fabsf(fxf) + fabsf(fyf)) * (size * iZ + 1.0f) * (1.0f + fabsf(qx) + fabsf(qy)) +
                        1e-6f * (fabsf(ux) + fabsf(uy) + fabsf(cxf) + fabsf(cyf));
        const float fw = (float)F.w, fh = (float)F.h;
        // (a depth within a thousand of its rounding errors says nothing in FP32)
        const bool deep = Z > 1e-4f * size;
        bool inside = deep && ux > -0.5f + e && ux < fw - 0.5f - e && uy > -0.5f + e && uy < fh - 0.5f - e;
        if (!inside && !(deep && (ux < -0.5f - e || ux > fw - 0.5f + e || uy < -0.5f - e || uy > fh - 0.5f + e))) {
          const double vw[3] = {(double)vx, (double)vy, (double)vz};
          double vc[3];
          mat3_vec_rn(F.R_wc, vw, vc);
#pragma unroll
          for (int i = 0; i < 3; ++i) vc[i] = __dadd_rn(vc[i], F.t_wc[i]);
          const long long pxi = llround(__dadd_rn(__ddiv_rn(__dmul_rn(F.fx, vc[0]), vc[2]), F.cx));
          const long long pyi = llround(__dadd_rn(__ddiv_rn(__dmul_rn(F.fy, vc[1]), vc[2]), F.cy));
          inside = pxi >= 0 && pxi < F.w && pyi >= 0 && pyi < F.h;
        }
        if (inside) {
          const int vox = (iz * F.ny + iy) * F.nx + ix;
          const unsigned int prev = atomicExch(&head[vox], r);
          rec[r] = make_uint2(prev, __float_as_uint(truncated_sdf(diff, trunc, F.inv_trunc)));
          if (prev == kNoRecord) voxel_of_first = vox;
        }
      }
    }
    first[(size_t)(s + F.steps) * npix + pix] = voxel_of_first;
  }
}

// One running-mean update (tsdf_fusion.cpp:95-102).
__device__ __forceinline__ void fold_update(float sdf, float w_new, float* t, float* w) {
  const float w_sum = __fadd_rn(*w, w_new);
  if (w_sum > 0.0f) {
    *t = __fdiv_rn(__fadd_rn(__fmul_rn(*w, *t), __fmul_rn(w_new, sdf)), w_sum);
    *w = w_sum;
  }
}

// A chain of up to N records from `last`, sorted in registers by an odd-even
// network and folded in ascending order.  False when the chain is longer.
template <int N>
__device__ __forceinline__ bool fold_short_chain(const uint2* rec, unsigned int last, float w_new, float* t,
                                                 float* w) {
  unsigned int key[N], i = last;
  float sdf[N];
#pragma unroll
  for (int j = 0; j < N; ++j) {
    key[j] = i;  // kNoRecord past the end: sorts last
    sdf[j] = 0.0f;
    if (i != kNoRecord) {
      const uint2 x = rec[i];
      sdf[j] = __uint_as_float(x.y);
      i = x.x;
    }
  }
  if (i != kNoRecord) return false;
#pragma unroll
  for (int round = 0; round < N; ++round)
#pragma unroll
    for (int j = round & 1; j + 1 < N; j += 2) {
      const bool swap = key[j] > key[j + 1];
      const unsigned int lo = swap ? key[j + 1] : key[j], hi = swap ? key[j] : key[j + 1];
      const float slo = swap ? sdf[j + 1] : sdf[j], shi = swap ? sdf[j] : sdf[j + 1];
      key[j] = lo;
      key[j + 1] = hi;
      sdf[j] = slo;
      sdf[j + 1] = shi;
    }
#pragma unroll
  for (int j = 0; j < N; ++j)
    if (key[j] != kNoRecord) fold_update(sdf[j], w_new, t, w);
  return true;
}

// Folds one voxel of up to kShortChain records: its chain back in the reference's
// order (ascending records) and into the running weighted mean.  The voxel's
// head is cleared for the next frame.  False, and nothing done, for a longer
// chain.
constexpr int kShortChain = 6;
__device__ __forceinline__ bool fold_voxel(int vox, unsigned int* head, const uint2* rec, float w_new, float* tsdf,
                                           float* weight) {
  float t = tsdf[vox], w = weight[vox];
  if (!fold_short_chain<kShortChain>(rec, head[vox], w_new, &t, &w)) return false;
  head[vox] = kNoRecord;
  tsdf[vox] = t;
  weight[vox] = w;
  return true;
}

// The voxels of a frame's chains, kFoldBlock records a block: the records that
// begin a chain (about one in three) are packed first, so that every lane of a
// warp follows a chain -- the kernel is bound by the latency of those dependent
// reads (38 % of the issue slots, 28 % of DRAM).  A frame touches the voxels it
// updates and no others: counting, scanning and folding over a whole 31 M voxel
// grid took 0.6 ms of a 1.3 ms frame; this takes 0.05 ms, and 0.01 ms for the
// long chains.
// Voxels with longer chains (one in two hundred at 1 mm and 640x480, where the
// mean is 2; nearly all of them from 4 mm) are listed for k_tsdf_fold_long.
constexpr int kFoldThreads = 256, kFoldBlock = 8 * kFoldThreads;
__global__ void __launch_bounds__(kFoldThreads) k_tsdf_fold(const int* __restrict__ first, unsigned int nrec,
                                                            unsigned int* head, const uint2* __restrict__ rec,
                                                            float w_new, float* tsdf, float* weight, int* longs,
                                                            unsigned int* num_long) {
  __shared__ int voxels[kFoldBlock];
  __shared__ int count;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  const unsigned int base = blockIdx.x * (unsigned int)kFoldBlock;
  const int lane = threadIdx.x & 31;
  int v[kFoldBlock / kFoldThreads];
#pragma unroll
  for (int j = 0; j < kFoldBlock / kFoldThreads; ++j) {
    const unsigned int r = base + j * kFoldThreads + threadIdx.x;
    v[j] = r < nrec && r >= base ? first[r] : -1;
  }
#pragma unroll
  for (int j = 0; j < kFoldBlock / kFoldThreads; ++j) {
    const unsigned int some = __ballot_sync(0xffffffffu, v[j] >= 0);
    int at = 0;
    if (lane == 0 && some) at = atomicAdd(&count, __popc(some));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (v[j] >= 0) voxels[at + __popc(some & ((1u << lane) - 1u))] = v[j];
  }
  __syncthreads();
  const int n = count;
  for (int i = threadIdx.x; i - lane < n; i += kFoldThreads) {  // whole warps
    const int vox = i < n ? voxels[i] : -1;
    const bool longer = vox >= 0 && !fold_voxel(vox, head, rec, w_new, tsdf, weight);
    const unsigned int some = __ballot_sync(0xffffffffu, longer);
    unsigned int at = 0;
    if (lane == 0 && some) at = atomicAdd(num_long, (unsigned int)__popc(some));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (longer) longs[at + __popc(some & ((1u << lane) - 1u))] = vox;
  }
}

// The long chains, a warp each.  A chain comes in the order of arrival, and its
// records have to be folded in ascending order.  Nothing is sorted: the walk
// marks each of its records in `mark` (the frame's `first` array, whose entries
// have all been used: [step][pixel], fully written by k_tsdf_walk, so no entry
// of an earlier frame is left in it) with a value that is this voxel's alone,
// and keeps the box of pixels and steps that they lie in.  The warp then reads
// the box in record order -- rows, columns, steps -- 128 entries at a time, and
// folds what carries the mark.  That is linear in the chain and in the box, which
// is about the voxel's projection; bound by the walk's dependent reads.  Relinking
// the chain in order, by one thread, was quadratic in it.  Two frames of 640x480
// and the extraction, all kernels: 1 mm 0.66 ms, 4 mm (40 records a voxel) 3.8
// -> 1.3 ms, 10 mm (300) 60.7 -> 1.6 ms, 50 mm 10.7 ms.
__global__ void __launch_bounds__(kFoldThreads) k_tsdf_fold_long(const int* __restrict__ longs,
                                                                 const unsigned int* __restrict__ num_long, int width,
                                                                 unsigned int npix, unsigned int nst, int* mark,
                                                                 unsigned int* head, const uint2* __restrict__ rec,
                                                                 float w_new, float* tsdf, float* weight) {
  constexpr int kEach = 4;  // entries a lane has in flight
  const unsigned int n = *num_long, w = (unsigned int)width;
  const unsigned int lane = threadIdx.x & 31, warps = gridDim.x * (kFoldThreads / 32);
  for (unsigned int k = blockIdx.x * (kFoldThreads / 32) + (threadIdx.x >> 5); k < n; k += warps) {
    const int vox = longs[k], tag = -2 - vox;  // below every voxel and the -1 of "no chain begins here"
    unsigned int u0 = 0xffffffffu, u1 = 0, v0 = 0xffffffffu, v1 = 0, s0 = 0xffffffffu, s1 = 0;
    for (unsigned int i = head[vox]; i != kNoRecord;) {
      const unsigned int next = rec[i].x;
      const unsigned int pix = i / nst, s = i - pix * nst, v = pix / w, u = pix - v * w;
      u0 = min(u0, u);
      u1 = max(u1, u);
      v0 = min(v0, v);
      v1 = max(v1, v);
      s0 = min(s0, s);
      s1 = max(s1, s);
      if (lane == 0) mark[(size_t)s * npix + pix] = tag;
      i = next;
    }
    __syncwarp();  // lane 0's marks before the other lanes' reads
    float t = tsdf[vox], wt = weight[vox];
    const unsigned int ns = s1 - s0 + 1u, row = (u1 - u0 + 1u) * ns;
    const unsigned long long all = (unsigned long long)(v1 - v0 + 1u) * row;  // at most the frame's records
    for (unsigned long long q0 = 0; q0 < all; q0 += 32 * kEach) {
      unsigned int r[kEach];
      bool hit[kEach];
#pragma unroll
      for (int j = 0; j < kEach; ++j) {
        const unsigned long long q = q0 + 32 * j + lane;
        hit[j] = q < all;
        r[j] = 0;
        if (hit[j]) {
          const unsigned int y = (unsigned int)q / row, in_row = (unsigned int)q - y * row;
          const unsigned int x = in_row / ns, s = s0 + (in_row - x * ns), pix = (v0 + y) * w + u0 + x;
          hit[j] = mark[(size_t)s * npix + pix] == tag;
          r[j] = pix * nst + s;
        }
      }
      float sdf[kEach];
#pragma unroll
      for (int j = 0; j < kEach; ++j) sdf[j] = hit[j] ? __uint_as_float(rec[r[j]].y) : 0.0f;
#pragma unroll
      for (int j = 0; j < kEach; ++j)
        for (unsigned int some = __ballot_sync(0xffffffffu, hit[j]); some; some &= some - 1u)
          fold_update(__shfl_sync(0xffffffffu, sdf[j], __ffs(some) - 1), w_new, &t, &wt);
    }
    if (lane == 0) {
      head[vox] = kNoRecord;
      tsdf[vox] = t;
      weight[vox] = wt;
    }
  }
}

constexpr unsigned kLongBlocks = 152 * 8;  // the warps that 152 SMs hold at once

__global__ void k_tsdf_fill(int64_t n, float* tsdf, float* weight) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  tsdf[i] = 1.0f;
  weight[i] = 0.0f;
}

// SurfaceGradient (tsdf_internal.h:154-187) at voxel (ix, iy, iz).
__device__ bool surface_gradient(const float* __restrict__ tsdf, const float* __restrict__ weight, int nx, int ny,
                                 int nz, int ix, int iy, int iz, float* onx, float* ony, float* onz) {
  const size_t i0 = ((size_t)iz * ny + iy) * nx + ix;
  if (weight[i0] <= 0.0f) return false;  // never fused
  if (tsdf[i0] > 0.0f) return false;
  const int off[6][3] = {{1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1}};
  float sx = 0.0f, sy = 0.0f, sz = 0.0f;
  bool pos = false;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int a = ix + off[k][0], b = iy + off[k][1], c = iz + off[k][2];
    if (!(a >= 0 && b >= 0 && c >= 0 && a < nx && b < ny && c < nz)) continue;
    const size_t j = ((size_t)c * ny + b) * nx + a;
    if (weight[j] > 0.0f && tsdf[j] > 0.0f) {
      pos = true;
      sx = __fadd_rn(sx, (float)off[k][0]);
      sy = __fadd_rn(sy, (float)off[k][1]);
      sz = __fadd_rn(sz, (float)off[k][2]);
    }
  }
  if (!pos) return false;
  const float len = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(sx, sx), __fmul_rn(sy, sy)), __fmul_rn(sz, sz)));
  if (len < 1e-9f) return false;
  *onx = __fdiv_rn(sx, len);
  *ony = __fdiv_rn(sy, len);
  *onz = __fdiv_rn(sz, len);
  return true;
}

// Surface voxels, kSurfaceBlock per block: bit i & 31 of mask[i / 32] and the
// block's count.  A pass over the weights (and over the distances of fused
// voxels only); the scan that places the points runs over the block counts.
// 31 M voxels: mask, scan and emit 0.12 ms, where flags, their scan over the
// grid and the emission took 0.55 ms and two more grids of memory.
constexpr int kSurfaceThreads = 256, kSurfaceBlock = 8 * kSurfaceThreads;
__global__ void __launch_bounds__(kSurfaceThreads) k_tsdf_surface_mask(const float* __restrict__ tsdf,
                                                                       const float* __restrict__ weight, int nx,
                                                                       int ny, int nz, unsigned int* mask,
                                                                       unsigned int* count) {
  const unsigned int n = (unsigned int)nx * ny * nz;  // below 2^31
  const unsigned int base = blockIdx.x * (unsigned int)kSurfaceBlock;
  constexpr int kEach = kSurfaceBlock / kSurfaceThreads;
  int mine = 0;
  float wt[kEach];
#pragma unroll
  for (int j = 0; j < kEach; ++j) {  // the block's weights, all in flight together
    const unsigned int i = base + j * kSurfaceThreads + threadIdx.x;
    wt[j] = i < n ? weight[i] : 0.0f;
  }
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const unsigned int i = base + j * kSurfaceThreads + threadIdx.x;
    bool hit = false;
    if (wt[j] > 0.0f && tsdf[i] <= 0.0f) {
      const int ix = (int)(i % nx), iy = (int)((i / nx) % ny), iz = (int)(i / ((unsigned int)nx * ny));
      float a, b, c;
      hit = surface_gradient(tsdf, weight, nx, ny, nz, ix, iy, iz, &a, &b, &c);
    }
    const unsigned int bits = __ballot_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31) == 0) mask[i >> 5] = bits;  // the array is padded to whole blocks
    mine += hit;
  }
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&total, mine);
  __syncthreads();
  if (threadIdx.x == 0) count[blockIdx.x] = (unsigned int)total;
}

// ExtractPoints (tsdf_fusion.cpp:106-140) in (iz, iy, ix) order: the
// surface voxels' centres (VoxelToWorld: FP64 origin + FP32 offset, rounded
// to FP32), normals, confidences min(1, weight / 64).  One block per
// kSurfaceBlock voxels: a warp takes every 8th mask word.
__global__ void __launch_bounds__(kSurfaceThreads) k_tsdf_surface_emit(
    const float* __restrict__ tsdf, const float* __restrict__ weight, int nx, int ny, int nz,
    const unsigned int* __restrict__ mask, const unsigned int* __restrict__ count,
    const unsigned int* __restrict__ offset, double ox, double oy, double oz, float voxel, double* pos, double* nrm,
    float* conf, int64_t* key) {
  constexpr int kWords = kSurfaceBlock / 32;
  static_assert(kWords == 64, "two words a lane below");
  const unsigned int b = blockIdx.x;
  if (count[b] == 0u) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // every warp: the words' exclusive prefix, words 2 lane and 2 lane + 1
  const uint2 mine = reinterpret_cast<const uint2*>(mask + (size_t)b * kWords)[lane];
  const unsigned int c0 = (unsigned int)__popc(mine.x), both = c0 + (unsigned int)__popc(mine.y);
  unsigned int before = both;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned int v = __shfl_up_sync(0xffffffffu, before, o);
    if (lane >= o) before += v;
  }
  before -= both;
  for (int j = warp; j < kWords; j += kSurfaceThreads / 32) {
    const unsigned int w0 = __shfl_sync(0xffffffffu, mine.x, j >> 1), w1 = __shfl_sync(0xffffffffu, mine.y, j >> 1);
    const unsigned int p0 = __shfl_sync(0xffffffffu, before, j >> 1), pc = __shfl_sync(0xffffffffu, c0, j >> 1);
    const unsigned int word = (j & 1) ? w1 : w0;
    if (!((word >> lane) & 1u)) continue;
    const unsigned int i = b * (unsigned int)kSurfaceBlock + (unsigned int)j * 32u + lane;
    const size_t k = (size_t)offset[b] + p0 + ((j & 1) ? pc : 0u) + __popc(word & ((1u << lane) - 1u));
    const int ix = (int)(i % nx), iy = (int)((i / nx) % ny), iz = (int)(i / ((unsigned int)nx * ny));
    float gx, gy, gz;
    surface_gradient(tsdf, weight, nx, ny, nz, ix, iy, iz, &gx, &gy, &gz);
    pos[3 * k + 0] = (double)__double2float_rn(__dadd_rn(ox, (double)__fmul_rn(__fadd_rn((float)ix, 0.5f), voxel)));
    pos[3 * k + 1] = (double)__double2float_rn(__dadd_rn(oy, (double)__fmul_rn(__fadd_rn((float)iy, 0.5f), voxel)));
    pos[3 * k + 2] = (double)__double2float_rn(__dadd_rn(oz, (double)__fmul_rn(__fadd_rn((float)iz, 0.5f), voxel)));
    nrm[3 * k + 0] = (double)gx;
    nrm[3 * k + 1] = (double)gy;
    nrm[3 * k + 2] = (double)gz;
    conf[k] = fminf(1.0f, __fdiv_rn(weight[i], 64.0f));
    key[k] = (int64_t)i;
  }
}

// FloorToIntScaled of the bounding-box extent + 1 (tsdf_fusion.cpp:36-47).
int grid_dim(double bbox_max, float origin, float voxel) {
  const int n = (int)floorf((float)(bbox_max - (double)origin) / voxel) + 1;
  return n > 1 ? n : 1;
}

}  // namespace

struct TsdfVolume {
  PoolUser pool_user;  // first, so that it goes last
  recon_tsdf_config cfg{};
  int device = 0;
  cudaStream_t stream = nullptr;
  int nx = 1, ny = 1, nz = 1;
  int64_t nvox = 1;
  float voxel = 0.0f;
  double origin[3] = {0, 0, 0};
  OwnArray<float> grid;         // tsdf, then weight
  OwnArray<unsigned int> head;  // per voxel its chain's latest record; kNoRecord between frames
  bool head_clean = false;      // false: a frame failed between filling chains and folding them
  // a frame's arrays, on the volume's stream
  PoolArray<uint16_t> depth;
  PoolArray<uint8_t> conf;
  PoolArray<uint2> rec;  // {previous record of the voxel, sdf bits}
  PoolArray<int> first;  // per record the voxel whose chain it begins, else -1
  PoolArray<double> tables;
  PoolArray<int> longs;  // the voxels with long chains
  PoolArray<unsigned int> scratch, counts;  // counts: {pixels integrated, long chains}
  TsdfVolume(int device_, cudaStream_t st)
      : device(device_), stream(st), depth(device_, st), conf(device_, st), rec(device_, st), first(device_, st),
        tables(device_, st), longs(device_, st), scratch(device_, st), counts(device_, st) {
    pool_user.join(device_);
  }
  float* tsdf() const { return grid.p; }
  float* weight() const { return grid.p + nvox; }
  void release() {
    grid.release();
    head.release();
    rec.release();
    first.release();
    depth.release();
    conf.release();
    tables.release();
    longs.release();
    scratch.release();
    counts.release();
  }
  ~TsdfVolume() {
    cudaSetDevice(device);
    release();
    if (stream) {
      cudaStreamSynchronize(stream);  // the pool's arrays are free when the volume is gone
      cudaStreamDestroy(stream);
    }
  }
};

}  // namespace rmvs

using namespace rmvs;

namespace {

recon_status tsdf_fail(recon_status st, const std::string& what) {
  g_last_error = what;
  return st;
}

recon_status cuda_fail(cudaError_t e, const char* what) {
  cudaGetLastError();
  g_last_error = std::string("tsdf: ") + what + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? RECON_ERR_OUT_OF_MEMORY : RECON_ERR_MVS_GPU_FAILURE;
}

#define TCK(call, what)                        \
  do {                                         \
    const cudaError_t e_ = (call);             \
    if (e_ != cudaSuccess) return cuda_fail(e_, what); \
  } while (0)

unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

extern "C" {

RECON_API recon_status recon_tsdf_config_default(recon_tsdf_config* out) {
  if (!out) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_config_default: NULL");
  std::memset(out, 0, sizeof(*out));
  out->voxel_size_m = 0.001;
  out->truncation_m = 0.008;
  out->min_depth_m = 0.05;
  out->max_depth_m = 3.0;
  out->fx = 1.0;
  out->fy = 1.0;
  out->bbox_max_x = 1.0;
  out->bbox_max_y = 1.0;
  out->bbox_max_z = 1.0;
  out->min_confidence = 30;
  return RECON_OK;
}

RECON_API recon_status recon_tsdf_create(const recon_tsdf_config* cfg, int32_t device, void** out_volume) {
  if (!cfg || !out_volume) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_create: NULL argument");
  *out_volume = nullptr;
  if (!(cfg->voxel_size_m > 0.0) || !(cfg->fx != 0.0) || !(cfg->fy != 0.0))
    return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_create: voxel size must be > 0 and focal lengths non-zero");
  const float voxel = (float)cfg->voxel_size_m;
  const double origin[3] = {(double)(float)cfg->origin_x, (double)(float)cfg->origin_y, (double)(float)cfg->origin_z};
  const int nx = grid_dim(cfg->bbox_max_x, (float)cfg->origin_x, voxel);
  const int ny = grid_dim(cfg->bbox_max_y, (float)cfg->origin_y, voxel);
  const int nz = grid_dim(cfg->bbox_max_z, (float)cfg->origin_z, voxel);
  if ((int64_t)nx * ny * nz >= (int64_t)1 << 31)
    return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_create: more than 2^31 voxels");
  cudaStream_t stream = nullptr;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) return cuda_fail(e, "create");
  auto* V = new (std::nothrow) TsdfVolume(device, stream);
  if (!V) {
    cudaStreamDestroy(stream);
    return tsdf_fail(RECON_ERR_OUT_OF_MEMORY, "tsdf_create: host allocation failed");
  }
  V->cfg = *cfg;
  V->voxel = voxel;
  for (int i = 0; i < 3; ++i) V->origin[i] = origin[i];
  V->nx = nx;
  V->ny = ny;
  V->nz = nz;
  V->nvox = (int64_t)nx * ny * nz;
  e = V->grid.reserve(2 * (size_t)V->nvox);
  if (e == cudaSuccess) {
    k_tsdf_fill<<<blocks_for(V->nvox, 256), 256, 0, V->stream>>>(V->nvox, V->tsdf(), V->weight());
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(V->stream);
  if (e != cudaSuccess) {
    const recon_status st = cuda_fail(e, "create");
    delete V;
    return st;
  }
  *out_volume = V;
  g_last_error.clear();
  return RECON_OK;
}

RECON_API recon_status recon_tsdf_integrate(void* volume, const uint16_t* depth_mm, const uint8_t* confidence,
                                            int32_t width, int32_t height, const double* world_to_camera,
                                            float depth_uncertainty_m, uint32_t* out_integrated) {
  if (out_integrated) *out_integrated = 0;
  if (!volume || !world_to_camera) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_integrate: NULL argument");
  TsdfVolume& V = *static_cast<TsdfVolume*>(volume);
  const recon_tsdf_config& c = V.cfg;
  // IntegrateFrame's early returns (tsdf_internal.h:50-54)
  if (!depth_mm || width <= 0 || height <= 0) return RECON_OK;
  const float trunc = (float)c.truncation_m;
  if (V.voxel <= 0.0f || trunc <= 0.0f) return RECON_OK;
  if ((int64_t)width * height > ((int64_t)1 << 26))
    return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_integrate: frame larger than 2^26 pixels");
  TsdfFrame F;
  std::memset(&F, 0, sizeof(F));
  F.w = width;
  F.h = height;
  F.nx = V.nx;
  F.ny = V.ny;
  F.nz = V.nz;
  F.voxel = V.voxel;
  F.trunc = trunc;
  F.steps = (int)(trunc / V.voxel) + 1;
  const double sig = (double)depth_uncertainty_m;
  const double sigma = sig > 1e-4 ? sig : 1e-4;
  F.w_new = (float)(1.0 / (sigma * sigma));
  F.fx = c.fx;
  F.fy = c.fy;
  F.cx = c.cx;
  F.cy = c.cy;
  F.min_depth = c.min_depth_m;
  F.max_depth = c.max_depth_m;
  F.min_conf = c.min_confidence;
  for (int i = 0; i < 3; ++i) F.origin[i] = V.origin[i];
  // R_cw = R_wc^T, t_cw = -(R_cw t_wc) (tsdf_internal.h:57-69), host FP64 in
  // the reference's order (this file is compiled without contractions)
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j) F.R_wc[i * 3 + j] = world_to_camera[i * 4 + j];
    F.t_wc[i] = world_to_camera[i * 4 + 3];
  }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) F.R_cw[j * 3 + i] = F.R_wc[i * 3 + j];
  for (int i = 0; i < 3; ++i) {
    double s = 0.0;
    for (int j = 0; j < 3; ++j) s += F.R_cw[i * 3 + j] * F.t_wc[j];
    F.t_cw[i] = -s;
  }
  TCK(cudaSetDevice(V.device), "set device");
  const size_t npix = (size_t)width * height;
  const int64_t nrec = (int64_t)npix * (2 * F.steps + 1);
  if (nrec >= ((int64_t)1 << 32)) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_integrate: too many updates");
  TCK(V.depth.reserve(npix), "alloc");
  if (confidence) TCK(V.conf.reserve(npix), "alloc");
  const size_t ntab = (size_t)width + height + V.nx + V.ny + V.nz;
  TCK(V.rec.reserve(nrec), "alloc");
  TCK(V.first.reserve(nrec), "alloc");
  TCK(V.tables.reserve(ntab), "alloc");
  TCK(V.longs.reserve((size_t)std::min<int64_t>(V.nvox, nrec / (kShortChain + 1))), "alloc");
  TCK(V.counts.reserve(2), "alloc");
  cudaStream_t st = V.stream;
  if (!V.head_clean) {
    TCK(V.head.reserve(V.nvox), "alloc");
    TCK(cudaMemsetAsync(V.head.p, 0xff, V.nvox * sizeof(unsigned int), st), "memset");
  }
  V.head_clean = false;
  F.inv_trunc = 1.0 / (double)trunc;
  F.r_scale = 1.0f;
  for (int i = 0; i < 9; ++i) {
    F.Rf[i] = (float)F.R_wc[i];
    F.r_scale = std::max(F.r_scale, std::fabs(F.Rf[i]));
  }
  for (int i = 0; i < 3; ++i) F.tf[i] = (float)F.t_wc[i];
  F.rotation = 1;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double dot = 0.0;
      for (int k = 0; k < 3; ++k) dot += F.R_wc[k * 3 + i] * F.R_wc[k * 3 + j];
      if (!(std::fabs(dot - (i == j ? 1.0 : 0.0)) <= 4e-16)) F.rotation = 0;
    }
  F.dir_x = V.tables.p;
  F.dir_y = F.dir_x + width;
  F.depth_of[0] = F.dir_y + height;
  F.depth_of[1] = F.depth_of[0] + V.nx;
  F.depth_of[2] = F.depth_of[1] + V.ny;
  TCK(cudaMemcpyAsync(V.depth.p, depth_mm, npix * sizeof(uint16_t), cudaMemcpyHostToDevice, st), "upload");
  if (confidence) TCK(cudaMemcpyAsync(V.conf.p, confidence, npix, cudaMemcpyHostToDevice, st), "upload");
  TCK(cudaMemsetAsync(V.counts.p, 0, 2 * sizeof(unsigned int), st), "memset");
  k_tsdf_tables<<<blocks_for((int64_t)ntab, 128), 128, 0, st>>>(F, V.tables.p);
  TCK(cudaGetLastError(), "tables");
  const dim3 b2(32, 8);
  k_tsdf_walk<<<dim3((width + 31) / 32, (height + 7) / 8), b2, 0, st>>>(
      F, V.depth.p, confidence ? V.conf.p : nullptr, V.head.p, V.rec.p, V.first.p, V.counts.p);
  TCK(cudaGetLastError(), "walk");
  k_tsdf_fold<<<blocks_for(nrec, kFoldBlock), kFoldThreads, 0, st>>>(V.first.p, (unsigned int)nrec, V.head.p, V.rec.p,
                                                                      F.w_new, V.tsdf(), V.weight(), V.longs.p,
                                                                      V.counts.p + 1);
  TCK(cudaGetLastError(), "fold");
  k_tsdf_fold_long<<<kLongBlocks, kFoldThreads, 0, st>>>(V.longs.p, V.counts.p + 1, width, (unsigned int)npix,
                                                         2u * F.steps + 1u, V.first.p, V.head.p, V.rec.p, F.w_new,
                                                         V.tsdf(), V.weight());
  TCK(cudaGetLastError(), "fold long");
  unsigned int n = 0;
  TCK(cudaMemcpyAsync(&n, V.counts.p, sizeof(n), cudaMemcpyDeviceToHost, st), "download");
  TCK(cudaStreamSynchronize(st), "integrate");
  V.head_clean = true;
  if (out_integrated) *out_integrated = n;
  g_last_error.clear();
  return RECON_OK;
}

RECON_API recon_status recon_tsdf_extract_points(void* volume, recon_mvs_point_cloud* out) {
  if (!volume || !out) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_extract_points: NULL argument");
  std::memset(out, 0, sizeof(*out));
  TsdfVolume& V = *static_cast<TsdfVolume*>(volume);
  TCK(cudaSetDevice(V.device), "set device");
  cudaStream_t st = V.stream;
  const unsigned int nblk = blocks_for(V.nvox, kSurfaceBlock);
  PoolArray<unsigned int> mask(V.device, st), count(V.device, st), offset(V.device, st);
  TCK(mask.reserve((size_t)nblk * (kSurfaceBlock / 32)), "alloc");
  TCK(count.reserve(nblk), "alloc");
  TCK(offset.reserve(nblk), "alloc");
  TCK(V.scratch.reserve(scan_scratch_elems(nblk)), "alloc");
  k_tsdf_surface_mask<<<nblk, kSurfaceThreads, 0, st>>>(V.tsdf(), V.weight(), V.nx, V.ny, V.nz, mask.p, count.p);
  TCK(cudaGetLastError(), "mask");
  TCK(exclusive_scan_u32(count.p, offset.p, nblk, V.scratch.p, st), "scan");
  unsigned int last_offset = 0, last_count = 0;
  TCK(cudaMemcpyAsync(&last_offset, offset.p + nblk - 1, sizeof(unsigned int), cudaMemcpyDeviceToHost, st), "download");
  TCK(cudaMemcpyAsync(&last_count, count.p + nblk - 1, sizeof(unsigned int), cudaMemcpyDeviceToHost, st), "download");
  TCK(cudaStreamSynchronize(st), "extract");
  const size_t n = (size_t)last_offset + last_count;
  if (n == 0) {
    g_last_error.clear();
    return RECON_OK;
  }
  PoolArray<double> pos(V.device, st), nrm(V.device, st);
  PoolArray<float> conf(V.device, st);
  PoolArray<int64_t> key(V.device, st);
  TCK(pos.reserve(3 * n), "alloc");
  TCK(nrm.reserve(3 * n), "alloc");
  TCK(conf.reserve(n), "alloc");
  TCK(key.reserve(n), "alloc");
  k_tsdf_surface_emit<<<nblk, kSurfaceThreads, 0, st>>>(V.tsdf(), V.weight(), V.nx, V.ny, V.nz, mask.p, count.p,
                                                        offset.p, V.origin[0], V.origin[1], V.origin[2], V.voxel,
                                                        pos.p, nrm.p, conf.p, key.p);
  TCK(cudaGetLastError(), "emit");
  out->count = (int64_t)n;
  out->positions = (double*)std::malloc(3 * sizeof(double) * n);
  out->normals = (double*)std::malloc(3 * sizeof(double) * n);
  out->colors = (float*)std::calloc(3 * n, sizeof(float));
  out->confidences = (float*)std::malloc(sizeof(float) * n);
  out->keys = (int64_t*)std::malloc(sizeof(int64_t) * n);
  out->counts = (uint32_t*)std::malloc(sizeof(uint32_t) * n);
  if (!out->positions || !out->normals || !out->colors || !out->confidences || !out->keys || !out->counts) {
    recon_mvs_point_cloud_free(out);
    return tsdf_fail(RECON_ERR_OUT_OF_MEMORY, "tsdf_extract_points: host allocation failed");
  }
  for (size_t i = 0; i < n; ++i) out->counts[i] = 1u;
  cudaError_t e = cudaMemcpyAsync(out->positions, pos.p, 3 * sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out->normals, nrm.p, 3 * sizeof(double) * n, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out->confidences, conf.p, sizeof(float) * n, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out->keys, key.p, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    recon_mvs_point_cloud_free(out);
    return cuda_fail(e, "extract download");
  }
  g_last_error.clear();
  return RECON_OK;
}

RECON_API recon_status recon_tsdf_dims(void* volume, int32_t* out_dims) {
  if (!volume || !out_dims) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_dims: NULL argument");
  const TsdfVolume& V = *static_cast<TsdfVolume*>(volume);
  out_dims[0] = V.nx;
  out_dims[1] = V.ny;
  out_dims[2] = V.nz;
  return RECON_OK;
}

RECON_API recon_status recon_tsdf_memory_usage(void* volume, uint64_t* out_bytes) {
  if (!volume || !out_bytes) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_memory_usage: NULL argument");
  const TsdfVolume& V = *static_cast<TsdfVolume*>(volume);
  *out_bytes = (uint64_t)V.nvox * 2 * sizeof(float);
  return RECON_OK;
}

RECON_API recon_status recon_tsdf_read_grid(void* volume, float* tsdf, float* weight) {
  if (!volume) return tsdf_fail(RECON_ERR_INVALID_ARGUMENT, "tsdf_read_grid: NULL volume");
  TsdfVolume& V = *static_cast<TsdfVolume*>(volume);
  TCK(cudaSetDevice(V.device), "set device");
  if (tsdf)
    TCK(cudaMemcpyAsync(tsdf, V.tsdf(), V.nvox * sizeof(float), cudaMemcpyDeviceToHost, V.stream), "download");
  if (weight)
    TCK(cudaMemcpyAsync(weight, V.weight(), V.nvox * sizeof(float), cudaMemcpyDeviceToHost, V.stream), "download");
  TCK(cudaStreamSynchronize(V.stream), "read grid");
  return RECON_OK;
}

RECON_API void recon_tsdf_destroy(void* volume) { delete static_cast<TsdfVolume*>(volume); }

}  // extern "C"
