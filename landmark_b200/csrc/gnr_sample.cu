// Ray generation, sampling + occupancy test, exclusive scan, compaction.
//
// Bit-exactness contract of the sampler: the set of valid (ray, sample) pairs equals what
// the torch renderer selects (sample_ray, app/models/gridnerf_sequential.py:260-281, then the
// alphaMask filter :460-465 with AlphaGridMask.sample_alpha, app/models/alpha_mask.py:35-59).
// Every floating-point operation below is therefore a single correctly rounded IEEE
// operation (__fadd_rn/__fmul_rn/__fdiv_rn are never contracted into FMAs), in the order
// in which torch's separate elementwise kernels apply them.
#include "gnr_internal.cuh"

namespace {

constexpr int kWarpsPerBlock = 8;

// ---------------------------------------------------------------------------------------------
// ray generation: d = (dir_x[i], dir_y[j], -1) @ R^T, o = c2w[:, 3]
// (dist_render/dataset/utils.py:57-89)
// ---------------------------------------------------------------------------------------------
struct Pose {
  float m[12];
};

__global__ void raygen_kernel(Pose pose, const float* __restrict__ dir_x, const float* __restrict__ dir_y,
                              int W, const int32_t* __restrict__ pixel_ids, int64_t first_pixel, int64_t n,
                              float* __restrict__ rays) {
  int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  int64_t pix = pixel_ids ? (int64_t)pixel_ids[r] : first_pixel + r;
  int j = (int)(pix / W), i = (int)(pix - (int64_t)j * W);
  float dx = dir_x[i], dy = dir_y[j], dz = -1.0f;
  float* out = rays + r * 6;
  out[0] = pose.m[3];
  out[1] = pose.m[7];
  out[2] = pose.m[11];
#pragma unroll
  for (int a = 0; a < 3; ++a)
    out[3 + a] = fmaf(dz, pose.m[a * 4 + 2], fmaf(dy, pose.m[a * 4 + 1], dx * pose.m[a * 4 + 0]));
}

// Same, with the pose read from device memory: a captured CUDA graph replays this launch for a new
// pose by rewriting those 12 floats.
__global__ void raygen_dev_kernel(const float* __restrict__ pose_dev, const float* __restrict__ dir_x,
                                  const float* __restrict__ dir_y, int W, const int32_t* __restrict__ pixel_ids,
                                  int64_t first_pixel, int64_t n, float* __restrict__ rays) {
  int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  float m[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) m[i] = __ldg(pose_dev + i);
  int64_t pix = pixel_ids ? (int64_t)pixel_ids[r] : first_pixel + r;
  int j = (int)(pix / W), i = (int)(pix - (int64_t)j * W);
  float dx = dir_x[i], dy = dir_y[j], dz = -1.0f;
  float* out = rays + r * 6;
  out[0] = m[3];
  out[1] = m[7];
  out[2] = m[11];
#pragma unroll
  for (int a = 0; a < 3; ++a) out[3 + a] = fmaf(dz, m[a * 4 + 2], fmaf(dy, m[a * 4 + 1], dx * m[a * 4 + 0]));
}

// ---------------------------------------------------------------------------------------------
// sampling: a warp per group of rays, 32 samples at a time
// ---------------------------------------------------------------------------------------------
// Continuous mask index of a coordinate: ((p - aabb0) * invgridSize - 1 + 1) / 2 * (size - 1), each operation rounded
// as torch rounds it.  The halving is exact, so it is folded into the last factor (`half` = (size - 1) / 2, exact too).
__device__ __forceinline__ float mask_index(float px, float lo, float inv, float half) {
  return __fmul_rn(__fadd_rn(gnr_normalize(px, lo, inv), 1.0f), half);
}

// AlphaGridMask.sample_alpha (app/models/alpha_mask.py:35-59): trilinear interpolation of the 0/1
// volume with zero padding, then `> threshold`.  The sum runs over the corners in grid_sample's
// order with individually rounded operations.  With a threshold of exactly zero the sum of
// non-negative weights is positive as soon as one occupied corner has a positive weight, so the
// loop can stop there.
__device__ __forceinline__ bool occupancy_corners(const GnrSampleParams& p, float ix, float iy, float iz) {
  // corners outside the volume contribute zero (padding_mode="zeros"); indices that do not
  // fit an int (only possible for samples far outside the mask box) are outside too.
  const bool okx = (ix >= -1.0f) && (ix < (float)p.aW), oky = (iy >= -1.0f) && (iy < (float)p.aH),
             okz = (iz >= -1.0f) && (iz < (float)p.aD);
  if (!(okx && oky && okz)) return 0.0f > p.a_thres;
  const float fx0 = floorf(ix), fy0 = floorf(iy), fz0 = floorf(iz);
  const int x0 = (int)fx0, y0 = (int)fy0, z0 = (int)fz0;
  const float fx1 = __fadd_rn(fx0, 1.0f), fy1 = __fadd_rn(fy0, 1.0f), fz1 = __fadd_rn(fz0, 1.0f);
  const float wx[2] = {__fsub_rn(fx1, ix), __fsub_rn(ix, fx0)};
  const float wy[2] = {__fsub_rn(fy1, iy), __fsub_rn(iy, fy0)};
  const float wz[2] = {__fsub_rn(fz1, iz), __fsub_rn(iz, fz0)};
  const bool stop_at_first = p.a_thres == 0.0f;
  float out = 0.0f;
#pragma unroll
  for (int cz = 0; cz < 2; ++cz) {
#pragma unroll
    for (int cy = 0; cy < 2; ++cy) {
      const int y = y0 + cy, z = z0 + cz;
      if ((unsigned)y >= (unsigned)p.aH || (unsigned)z >= (unsigned)p.aD) continue;
      const uint32_t row = (uint32_t)((z * p.aH + y) * p.aW);
#pragma unroll
      for (int cx = 0; cx < 2; ++cx) {
        const int x = x0 + cx;
        if ((unsigned)x < (unsigned)p.aW) {
          const uint32_t bit = row + (uint32_t)x;
          if ((__ldg(p.a_bits + (bit >> 5)) >> (bit & 31)) & 1u) {
            const float w = __fmul_rn(__fmul_rn(wx[cx], wy[cy]), wz[cz]);
            out = __fadd_rn(out, w);  // tap is exactly 1, so tap * w == w
            if (stop_at_first && w > 0.0f) return true;
          }
        }
      }
    }
  }
  return out > p.a_thres;
}

// floor of 0 <= x < 2^22 as a float and an int with two full-rate additions: rounding towards minus infinity at
// 2^23 leaves the integer part in the low mantissa bits.
__device__ __forceinline__ float floor_small(float x, int& i) {
  const float m = __fadd_rd(x, 8388608.0f);
  i = __float_as_int(m) & 0x7fffff;
  return __fsub_rn(m, 8388608.0f);
}

__device__ __forceinline__ bool occupancy_test(const GnrSampleParams& p, float px, float py, float pz) {
  const float ix = mask_index(px, p.a_lo[0], p.a_inv[0], p.a_half[0]);
  const float iy = mask_index(py, p.a_lo[1], p.a_inv[1], p.a_half[1]);
  const float iz = mask_index(pz, p.a_lo[2], p.a_inv[2], p.a_half[2]);
  if (p.a_thres == 0.0f && fminf(fminf(ix, iy), iz) > 0.0f && ix < p.a_end[0] && iy < p.a_end[1] &&
      iz < p.a_end[2]) {
    int x0, y0, z0;
    const float fx = floor_small(ix, x0), fy = floor_small(iy, y0), fz = floor_small(iz, z0);
    // strictly inside a cell all eight corner weights are positive (differences of floats that are not equal; their
    // product is far above the smallest float), so the sum is positive exactly if one of the corners is occupied
    if (fx != ix && fy != iy && fz != iz) {
      const uint32_t bit = ((uint32_t)z0 * (uint32_t)p.aH + (uint32_t)y0) * (uint32_t)p.aW + (uint32_t)x0;
      return (__ldg(p.a_any8 + (bit >> 5)) >> (bit & 31)) & 1u;
    }
  }
  return occupancy_corners(p, ix, iy, iz);
}

struct RaySetup {  // what the sample tests need of a ray, in shared memory
  float o[3], t_min, d[3], pad;
};

// What the two ends of a run prove about all its samples k0 .. k1: 0 = none is valid, 1 = all are, 2 = still open.
// fl(t_min + fl(step k)), the point, and the mask index are each monotone in their argument (every operation is a
// correctly rounded monotone function), so along each axis every sample between the two end samples lies between them,
// without any tolerance: if both are inside the box all are, if both are outside on the same side none is, and the mask
// cells of all samples lie in the range spanned by the cells of the two.  The hull sampler's distance is a_k + far u_k
// with a_k and u_k from the caller's tables: the run lies between the sums of the terms' smallest and of their largest
// values, whatever the order of the tables (their ranges over runs and words are kept beside them).  For
// a_k = near (1 - u_k), rising u_k and a near distance of 0.05 that is hardly wider than the two end samples.
// BLOCKS: the occupancy of that range is looked up in blocks of 2x2x2 cells, else cell by cell; a run that spans more
// than four of either along an axis stays open.  (Blocks of 4x4x4 cells, two at most, left 55 % of a city frame's words
// open; 22 % is what mixes valid and other samples.)
template <bool BLOCKS>
__device__ __forceinline__ int run_by_ends(const GnrSampleParams& p, const RaySetup& r, int k0, int k1) {
  float t0, t1;
  if (p.mode == 0) {
    t0 = gnr_sample_t(p, r.t_min, k0);
    t1 = gnr_sample_t(p, r.t_min, k1);
  } else {
    if (!(fabsf(r.t_min) < 1e30f)) return 2;  // (far u_k is not monotone where 0 x inf comes up)
    const float4 range = __ldg(p.hull_ranges + (BLOCKS ? (p.S + 7) / 8 + k0 / 32 : k0 / 8));
    const float f0 = __fmul_rn(r.t_min, range.z), f1 = __fmul_rn(r.t_min, range.w);
    t0 = __fadd_rn(range.x, fminf(f0, f1));
    t1 = __fadd_rn(range.y, fmaxf(f0, f1));
    if (!(t0 <= t1)) return 2;
  }
  float q0[3], q1[3];
  bool in = true;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    q0[a] = gnr_point(r.o[a], r.d[a], t0);
    q1[a] = gnr_point(r.o[a], r.d[a], t1);
    const float lo = fminf(q0[a], q1[a]), hi = fmaxf(q0[a], q1[a]);
    if (hi < p.lo[a] || lo > p.hi[a]) return 0;
    in = in && !(p.lo[a] > lo) && !(hi > p.hi[a]);
  }
  if (!in) return 2;
  if (!p.has_mask) return 1;
  if (!(p.a_thres >= 0.0f)) return 2;
  int b0[3], b1[3];
  const int size[3] = {p.aW, p.aH, p.aD};
  bool inside_cell = true;  // all samples strictly inside one cell
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float i0 = mask_index(q0[a], p.a_lo[a], p.a_inv[a], p.a_half[a]), i1 = mask_index(q1[a], p.a_lo[a], p.a_inv[a], p.a_half[a]);
    const float lo = fminf(i0, i1), hi = fmaxf(i0, i1);
    if (!(lo >= 0.0f && hi < (float)size[a])) return 2;
    b0[a] = (int)lo;
    b1[a] = (int)hi;
    if (BLOCKS) {
      b0[a] >>= 1;
      b1[a] >>= 1;
    } else {
      inside_cell = inside_cell && b0[a] == b1[a] && (float)b0[a] != lo;
    }
    if (b1[a] - b0[a] > 3) return 2;
  }
  const uint32_t nx = (uint32_t)(BLOCKS ? p.cW : p.aW), ny = (uint32_t)(BLOCKS ? p.cH : p.aH);
  const uint32_t* any_bits = BLOCKS ? p.a_coarse : p.a_any8;
  const uint32_t* all_bits = BLOCKS ? p.a_full : p.a_bits;
  const uint32_t row_bits = (2u << (b1[0] - b0[0])) - 1u;  // the range along x: at most four neighbouring bits
  uint32_t any = 0u, miss = 0u;
  for (int z = b0[2]; z <= b1[2]; ++z)
    for (int y = b0[1]; y <= b1[1]; ++y) {
      const uint32_t at = ((uint32_t)z * ny + (uint32_t)y) * nx + (uint32_t)b0[0], word = at >> 5, s = at & 31u;
      uint32_t a = __ldg(any_bits + word) >> s, f = __ldg(all_bits + word) >> s;
      if (row_bits >> (31u - s) > 1u) {  // (the row goes on in the next word)
        a |= __ldg(any_bits + word + 1) << (32u - s);
        f |= __ldg(all_bits + word + 1) << (32u - s);
      }
      any |= a & row_bits;
      miss |= ~f & row_bits;
    }
  const bool all = miss == 0u && p.a_thres == 0.0f;
  // no occupied corner in reach: the sum is zero.  Threshold zero: with its lower corner occupied a sample has a positive
  // weight, (x0 + 1 - ix)(y0 + 1 - iy)(z0 + 1 - iz), wherever in the cell it lies; strictly inside a cell any corner will do
  if (any == 0u) return 0;
  if (!BLOCKS && inside_cell && p.a_thres == 0.0f) return 1;
  return all ? 1 : 2;
}

__device__ __forceinline__ bool sample_valid(const GnrSampleParams& p, const RaySetup& r, int k) {
  const float t = gnr_sample_t(p, r.t_min, k);
  const float px = gnr_point(r.o[0], r.d[0], t), py = gnr_point(r.o[1], r.d[1], t), pz = gnr_point(r.o[2], r.d[2], t);
  const bool lo_out = (p.lo[0] > px) | (p.lo[1] > py) | (p.lo[2] > pz);
  const bool hi_out = (px > p.hi[0]) | (py > p.hi[1]) | (pz > p.hi[2]);
  return !(lo_out | hi_out) && (!p.has_mask || occupancy_test(p, px, py, pz));
}

constexpr int kSampleWarps = 4;

// A warp takes `per_warp` consecutive rays.  It sets them up one ray per lane, then walks their validity words, 32 words
// (of one or several rays) at a time, in three steps: every lane tries to decide its own word from the word's two end
// samples; the words that stay open are cut into runs of eight samples, 32 runs at a time, and decided the same way cell
// by cell; the runs that stay open are tested sample by sample, four runs at a time.  Each step queues what it leaves
// open in shared memory, so that the lanes of the next one are full.
// Bound by instruction issue.  A ray's latency is a few passes instead of one dependent step per sample, and most samples
// are never looked at: of a city frame's words 22 % stay open after the first step and 0.9 runs of each after the second.
// 131,072 rays x 384 samples (12 words a ray): 89 us, 38 warp instructions per word (119 us with first-step blocks of
// 4x4x4 cells, which left 55 % of the words open); 333 rays x 128 samples: 14 us, 121 us with a thread walking each ray.
__global__ void __launch_bounds__(kSampleWarps * 32, 8)
sample_words_kernel(const __grid_constant__ GnrSampleParams p, const float* __restrict__ rays, int64_t n_rays, int per_warp,
                    float* __restrict__ t_min_out, uint32_t* __restrict__ words_out, int32_t* __restrict__ counts_out,
                    int32_t* __restrict__ status) {
  if (status != nullptr && blockIdx.x == 0 && threadIdx.x < GNR_ST_WORDS) status[threadIdx.x] = 0;
  __shared__ RaySetup s_ray[kSampleWarps][32];
  __shared__ int s_count[kSampleWarps][32];
  __shared__ uint32_t s_bits[kSampleWarps][32];   // the 32 words of a pass
  __shared__ uint32_t s_item[kSampleWarps][32];   // ray << 16 | word of each of them
  __shared__ uint8_t s_open[kSampleWarps][32];    // open words: number in the pass
  __shared__ uint8_t s_run[kSampleWarps][128];    // open runs: number in the pass << 2 | run
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t below = (1u << lane) - 1u;
  const int64_t first = ((int64_t)blockIdx.x * kSampleWarps + warp) * per_warp;
  if (first >= n_rays) return;
  const int mine = (int)min((int64_t)per_warp, n_rays - first);
  if (lane < mine) {
    const float* r = rays + (first + lane) * 6;
    RaySetup s;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s.o[a] = __ldg(r + a);
      s.d[a] = __ldg(r + 3 + a);
    }
    // slab entry: max over axes of min(rate_a, rate_b), clamped to [near, far]
    float t_min = -INFINITY;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float vec = (s.d[a] == 0.0f) ? 1e-6f : s.d[a];
      const float ra = __fdiv_rn(__fsub_rn(p.hi[a], s.o[a]), vec);
      const float rb = __fdiv_rn(__fsub_rn(p.lo[a], s.o[a]), vec);
      t_min = fmaxf(t_min, fminf(ra, rb));
    }
    t_min = fminf(fmaxf(t_min, p.near_t), p.far_t);
    if (p.mode == 1) {
      // hull sampler: the per-ray parameter is `far`, the hit with the ground plane z = aabb_min_z
      // (far = -(o_z - z0) / d_z, replaced by near_far[1] for rays that do not point down)
      const float far = -__fdiv_rn(__fsub_rn(s.o[2], p.lo[2]), s.d[2]);
      t_min = (s.d[2] >= 0.0f) ? p.far_t : far;
    }
    s.t_min = t_min;
    s.pad = 0.0f;
    s_ray[warp][lane] = s;
    s_count[warp][lane] = 0;
    t_min_out[first + lane] = t_min;
  }
  __syncwarp();
  const int W = p.words, items = mine * W;
  int ray = lane / W, word = lane - ray * W;  // this lane's item: word `word` of ray `ray` of the warp
  const int ray_step = 32 / W, word_step = 32 - ray_step * W;
  for (int i0 = 0; i0 < items; i0 += 32) {
    const bool has = i0 + lane < items;
    int verdict = 0;
    if (has) verdict = run_by_ends<true>(p, s_ray[warp][ray], 32 * word, min(32 * word + 31, p.S - 1));
    const uint32_t open = __ballot_sync(0xffffffffu, verdict == 2);
    s_bits[warp][lane] = verdict != 1 ? 0u : (p.S - 32 * word >= 32 ? 0xffffffffu : (1u << (p.S - 32 * word)) - 1u);
    s_item[warp][lane] = ((uint32_t)ray << 16) | (uint32_t)word;
    if (verdict == 2) s_open[warp][__popc(open & below)] = (uint8_t)lane;
    __syncwarp();
    const int n_open = __popc(open);
    int n_run = 0;
    for (int j0 = 0; j0 < 4 * n_open; j0 += 32) {  // lane = run of eight samples
      const int j = j0 + lane;
      int v = 0, at = 0, run = j & 3;
      if (j < 4 * n_open) {
        at = s_open[warp][j >> 2];
        const uint32_t it = s_item[warp][at];
        const int k = 32 * (int)(it & 0xffffu) + 8 * run;
        if (k < p.S) {
          v = run_by_ends<false>(p, s_ray[warp][it >> 16], k, min(k + 7, p.S - 1));
          if (v == 1) atomicOr(&s_bits[warp][at], (k + 8 <= p.S ? 0xffu : (1u << (p.S - k)) - 1u) << (8 * run));
        }
      }
      const uint32_t still = __ballot_sync(0xffffffffu, v == 2);
      if (v == 2) s_run[warp][n_run + __popc(still & below)] = (uint8_t)(at << 2 | run);
      n_run += __popc(still);
    }
    __syncwarp();
    for (int j0 = 0; j0 < n_run; j0 += 4) {  // lane = sample
      const int j = j0 + (lane >> 3);
      bool valid = false;
      int at = 0, run = 0;
      if (j < n_run) {
        const int e = s_run[warp][j];
        at = e >> 2;
        run = e & 3;
        const uint32_t it = s_item[warp][at];
        const int k = 32 * (int)(it & 0xffffu) + 8 * run + (lane & 7);
        valid = k < p.S && sample_valid(p, s_ray[warp][it >> 16], k);
      }
      const uint32_t vote = __ballot_sync(0xffffffffu, valid);
      const uint32_t byte = (vote >> (lane & 24)) & 0xffu;
      if ((lane & 7) == 0 && byte) atomicOr(&s_bits[warp][at], byte << (8 * run));
    }
    __syncwarp();
    if (has) {
      const uint32_t bits = s_bits[warp][lane];
      words_out[first * W + i0 + lane] = bits;
      if (bits) atomicAdd(&s_count[warp][ray], __popc(bits));
    }
    ray += ray_step;
    word += word_step;
    if (word >= W) {
      word -= W;
      ++ray;
    }
    __syncwarp();
  }
  if (lane < mine) counts_out[first + lane] = s_count[warp][lane];
}

// ---------------------------------------------------------------------------------------------
// exclusive scan of int32 (three small kernels, no inter-block waits)
// ---------------------------------------------------------------------------------------------
constexpr int kScanBlock = 1024;

__device__ __forceinline__ int block_exclusive_scan(int v, int* total) {
  __shared__ int warp_sums[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int s = warp_sums[lane];
    int si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += t;
    }
    warp_sums[lane] = si - s;  // exclusive warp base
    if (lane == 31) *total = si;
  }
  __syncthreads();
  int res = warp_sums[wid] + incl - v;
  __syncthreads();
  return res;
}

__global__ void __launch_bounds__(kScanBlock)
scan_local_kernel(const int32_t* __restrict__ in, int32_t* __restrict__ out, int32_t* __restrict__ block_sums, int64_t n) {
  __shared__ int total;
  int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  int v = (i < n) ? in[i] : 0;
  int ex = block_exclusive_scan(v, &total);
  if (i < n) out[i] = ex;
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanBlock)
scan_sums_kernel(int32_t* __restrict__ block_sums, int n_blocks, int32_t* __restrict__ out_total,
                 int32_t* __restrict__ status, int total_slot, int overflow_slot, long long capacity) {
  __shared__ int total;
  long long carry = 0;
  for (int base = 0; base < n_blocks; base += kScanBlock) {
    int i = base + threadIdx.x;
    int v = (i < n_blocks) ? block_sums[i] : 0;
    int ex = block_exclusive_scan(v, &total);
    if (i < n_blocks) block_sums[i] = (int)(carry + ex);
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *out_total = (int)carry;
    status[total_slot] = (int)carry;
    status[overflow_slot] = (carry > capacity) ? 1 : 0;
  }
}

__global__ void __launch_bounds__(kScanBlock)
scan_add_kernel(int32_t* __restrict__ out, const int32_t* __restrict__ block_sums, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  if (i < n) out[i] += block_sums[blockIdx.x];
}

// ---------------------------------------------------------------------------------------------
// compaction: ids[offsets[ray] + rank of sample among the ray's valid ones] = ray << kbits | k
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
expand_ids_kernel(const uint32_t* __restrict__ words, const int32_t* __restrict__ offsets, int64_t n_rays, int n_words,
                  int kbits, long long capacity, uint32_t* __restrict__ ids) {
  const int lane = threadIdx.x & 31;
  int64_t ray = (int64_t)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (ray >= n_rays) return;
  long long pos = offsets[ray];
  long long end = offsets[ray + 1];
  if (pos == end) return;
  const uint32_t* wrow = words + ray * n_words;
  for (int w = 0; w < n_words && pos < end; ++w) {
    uint32_t bits = __ldg(wrow + w);
    if ((bits >> lane) & 1u) {
      long long at = pos + __popc(bits & ((1u << lane) - 1u));
      if (at < capacity) ids[at] = ((uint32_t)ray << kbits) | (uint32_t)(w * 32 + lane);
    }
    pos += __popc(bits);
  }
}

}  // namespace

int launch_exclusive_scan(const int32_t* counts, int32_t* offsets, int32_t* block_sums, int64_t n,
                          int32_t* status, int total_slot, int overflow_slot, int64_t capacity,
                          cudaStream_t st) {
  int n_blocks = (int)((n + kScanBlock - 1) / kScanBlock);
  if (n_blocks < 1) n_blocks = 1;
  scan_local_kernel<<<n_blocks, kScanBlock, 0, st>>>(counts, offsets, block_sums, n);
  scan_sums_kernel<<<1, kScanBlock, 0, st>>>(block_sums, n_blocks, offsets + n, status, total_slot, overflow_slot,
                                             (long long)capacity);
  scan_add_kernel<<<n_blocks, kScanBlock, 0, st>>>(offsets, block_sums, n);
  return (int)cudaGetLastError();
}

// Rays per warp: up to 32 (the slab set-up then uses every lane), as few as fill whole waves of the 32 warps an SM holds:
// rounded down, one ray a warp for 8192 rays made 1.7 waves (146.3 us per fp32 call against 141.5), and 27 for 131,072
// rays 30 blocks more than the GPU holds at a time (1890 against 1884 us for 518,400 rays).
static int launch_sample_words(const GnrModel* m, const GnrSampleParams& p, const float* rays, int64_t n, float* t_min,
                               uint32_t* words, int32_t* counts, cudaStream_t st, int32_t* status = nullptr) {
  const int64_t warps = (int64_t)m->sm_count * 32, waves = (n + 32 * warps - 1) / (32 * warps);
  const int per_warp = (int)((n + waves * warps - 1) / (waves * warps));
  const int64_t per_block = (int64_t)per_warp * kSampleWarps;
  sample_words_kernel<<<(unsigned)((n + per_block - 1) / per_block), kSampleWarps * 32, 0, st>>>(p, rays, n, per_warp, t_min, words,
                                                                                               counts, status);
  return (int)cudaGetLastError();
}

int launch_sample_mask(const GnrModel* m, const GnrSampleParams& p, const float* rays, int64_t n, char* ws,
                       const GnrWs& L, cudaStream_t st, int32_t* status) {
  return launch_sample_words(m, p, rays, n, (float*)(ws + L.t_min), (uint32_t*)(ws + L.words), (int32_t*)(ws + L.counts), st,
                             status);
}

int launch_sample_compact(const GnrModel* m, const GnrSampleParams& p, int64_t n, char* ws, const GnrWs& L,
                          int64_t max_valid, int with_ids, cudaStream_t st) {
  (void)m;
  int32_t* offsets = (int32_t*)(ws + L.offsets);
  int e = launch_exclusive_scan((const int32_t*)(ws + L.counts), offsets, (int32_t*)(ws + L.block_sums), n,
                                (int32_t*)(ws + L.status), GNR_ST_NUM_VALID, GNR_ST_OVERFLOW_VALID, max_valid, st);
  if (e || !with_ids) return e;  // the fused march pass and the appearance compaction read the words themselves
  unsigned blocks = (unsigned)((n + kWarpsPerBlock - 1) / kWarpsPerBlock);
  expand_ids_kernel<<<blocks, kWarpsPerBlock * 32, 0, st>>>((const uint32_t*)(ws + L.words), offsets, n, p.words, p.kbits,
                                                           (long long)max_valid, (uint32_t*)(ws + L.ids));
  return (int)cudaGetLastError();
}

extern "C" int gnr_generate_rays(const float* pose_h, const float* dir_x, const float* dir_y, int H, int W,
                                 const int32_t* pixel_ids, int64_t first_pixel, int64_t n, float* rays,
                                 void* stream) {
  if (!pose_h || !dir_x || !dir_y || !rays || H <= 0 || W <= 0 || n < 0) {
    gnr_set_error("gnr_generate_rays: bad argument");
    return -1;
  }
  if (!pixel_ids && (first_pixel < 0 || first_pixel + n > (int64_t)H * W)) {
    gnr_set_error("gnr_generate_rays: pixel range [%lld, %lld) outside the %dx%d image", (long long)first_pixel,
                  (long long)(first_pixel + n), W, H);
    return -1;
  }
  if (n == 0) return 0;
  Pose p;
  for (int i = 0; i < 12; ++i) p.m[i] = pose_h[i];
  raygen_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(p, dir_x, dir_y, W, pixel_ids,
                                                                              first_pixel, n, rays);
  GNR_CUDA_OK(cudaGetLastError());
  return 0;
}

extern "C" int gnr_generate_rays_dev(const float* pose_dev, const float* dir_x, const float* dir_y, int H, int W,
                                     const int32_t* pixel_ids, int64_t first_pixel, int64_t n, float* rays,
                                     void* stream) {
  if (!pose_dev || !dir_x || !dir_y || !rays || H <= 0 || W <= 0 || n < 0) {
    gnr_set_error("gnr_generate_rays_dev: bad argument");
    return -1;
  }
  if (!pixel_ids && (first_pixel < 0 || first_pixel + n > (int64_t)H * W)) {
    gnr_set_error("gnr_generate_rays_dev: pixel range [%lld, %lld) outside the %dx%d image", (long long)first_pixel,
                  (long long)(first_pixel + n), W, H);
    return -1;
  }
  if (n == 0) return 0;
  raygen_dev_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(pose_dev, dir_x, dir_y, W, pixel_ids,
                                                                                  first_pixel, n, rays);
  GNR_CUDA_OK(cudaGetLastError());
  return 0;
}

// ---------------------------------------------------------------------------------------------
// Allocation-free sampling: same kernels, scratch in a fixed device array of this library.
// ---------------------------------------------------------------------------------------------
// Scratch of gnr_sample_static: [validity bit words][scan block sums].  One copy per GPU that
// loads the library, shared by every call on that GPU.
static __device__ __align__(256) unsigned char g_sample_static_scratch[GNR_SAMPLE_STATIC_SCRATCH_BYTES];

#include <mutex>

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mutex;
unsigned char* g_static_ptr[kMaxDevices] = {nullptr};

// Device address of the scratch array on `device`.  The array's name is only a host-side
// handle; the address a kernel can use comes from cudaGetSymbolAddress, asked once per
// device with that device current.
int static_scratch_for(int device, unsigned char** out) {
  if (device < 0 || device >= kMaxDevices) {
    gnr_set_error("gnr_sample_static: device ordinal %d outside [0, %d)", device, kMaxDevices);
    return -1;
  }
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (!g_static_ptr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_sample_static_scratch);
    if (e != cudaSuccess || !p) {
      gnr_set_error("gnr_sample_static: cudaGetSymbolAddress failed on device %d: %s", device, cudaGetErrorString(e));
      return -2;
    }
    g_static_ptr[device] = (unsigned char*)p;
  }
  *out = g_static_ptr[device];
  return 0;
}

inline size_t round256(size_t v) { return (v + 255) / 256 * 256; }
}  // namespace

extern "C" int gnr_sample_static(GnrModel* m, const float* rays, int64_t n_rays, int n_samples, int64_t max_valid,
                                 float* t_min, int32_t* counts, int32_t* offsets, uint32_t* ids, int32_t* status,
                                 void* stream) {
  if (!m) {
    gnr_set_error("gnr_sample_static: null model");
    return -1;
  }
  if (!rays || !t_min || !counts || !offsets || !ids || !status) {
    gnr_set_error("gnr_sample_static: rays and all five output buffers are required");
    return -1;
  }
  if (n_rays < 1 || n_samples < 1 || max_valid < 1) {
    gnr_set_error("gnr_sample_static: bad sizes (n_rays %lld, n_samples %d, max_valid %lld)", (long long)n_rays, n_samples,
                  (long long)max_valid);
    return -1;
  }
  // the same sampler preconditions gnr_sample checks (hull tables present and of this length)
  if (gnr_check_sampler(m, n_samples)) return -1;
  const int kbits = gnr_sample_bits(n_samples);
  if (kbits > 20 || n_rays > ((int64_t)1 << (32 - kbits)) || n_rays * (int64_t)n_samples > 0x7fffffffLL ||
      max_valid > 0x7fffffffLL) {
    gnr_set_error("gnr_sample_static: %lld rays x %d samples does not fit the 32-bit sample ids", (long long)n_rays, n_samples);
    return -1;
  }
  const size_t words = (size_t)(n_samples + 31) / 32;
  const size_t words_bytes = round256((size_t)n_rays * words * 4);
  const size_t sums_bytes = round256(((size_t)n_rays / 1024 + 2) * 4);
  if (words_bytes + sums_bytes > (size_t)GNR_SAMPLE_STATIC_SCRATCH_BYTES) {
    gnr_set_error("gnr_sample_static: %lld rays x %d samples need %zu bytes of scratch, the built-in array holds %u; "
                  "split the chunk or use gnr_sample with a workspace",
                  (long long)n_rays, n_samples, words_bytes + sums_bytes, (unsigned)GNR_SAMPLE_STATIC_SCRATCH_BYTES);
    return -1;
  }
  int prev = 0;
  cudaGetDevice(&prev);
  if (prev != m->device) cudaSetDevice(m->device);
  unsigned char* scratch = nullptr;
  int rc = static_scratch_for(m->device, &scratch);
  if (rc == 0) {
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* mask_words = (uint32_t*)scratch;
    int32_t* block_sums = (int32_t*)(scratch + words_bytes);
    GnrSampleParams p = gnr_sample_params(m, n_samples);
    const unsigned blocks = (unsigned)((n_rays + kWarpsPerBlock - 1) / kWarpsPerBlock);
    cudaError_t e = cudaMemsetAsync(status, 0, GNR_ST_WORDS * sizeof(int32_t), st);  // the overflow flag starts at zero
    if (e == cudaSuccess) {
      // every word of mask_words and block_sums that is read below is written first by these
      // launches, so what an earlier call left in the array is never seen
      e = (cudaError_t)launch_sample_words(m, p, rays, n_rays, t_min, mask_words, counts, st);
    }
    if (e == cudaSuccess) {
      e = (cudaError_t)launch_exclusive_scan(counts, offsets, block_sums, n_rays, status, GNR_ST_NUM_VALID,
                                             GNR_ST_OVERFLOW_VALID, max_valid, st);
    }
    if (e == cudaSuccess) {
      expand_ids_kernel<<<blocks, kWarpsPerBlock * 32, 0, st>>>(mask_words, offsets, n_rays, p.words, p.kbits,
                                                               (long long)max_valid, ids);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
      gnr_set_error("gnr_sample_static: launch failed: %s", cudaGetErrorString(e));
      rc = -2;
    }
  }
  if (prev != m->device) cudaSetDevice(prev);
  return rc;
}
