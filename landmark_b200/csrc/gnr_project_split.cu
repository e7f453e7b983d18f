// Appearance gather from fp32 planes and lines + basis projection, the projection on the tensor cores with operands as
// sums of 16-bit terms (gnr_split.cuh): mlp_mode 0, and mlp_mode 1 with up to 152 products per sample.
//
// compute_appfeature (app/models/gridnerf_sequential.py:829-871).  The plane x line products are computed in fp32 as
// app_gather_kernel computes them (operations and order); app_dim x (pairs x channels) multiply-adds per sample follow,
// which on the CUDA cores cost more than the gather (their weights come through the same L1 / shared-memory port as the
// texels).
//
// One persistent CTA per SM, tiles of 128 samples (row = lane of tensor memory).  Sixteen warps gather: two groups of 256
// threads, two per row, take alternate tiles; each thread interpolates half the channels of a pair, eight at a time (six
// 256-bit loads), splits the products and stores them into a slot of a ring in tensor memory (one slot per pair, six
// slots: two tiles of the usual three pairs).
// A gatherer waits for its slot by the parity of the slot's use, which one bit tells apart only while the use before the
// last is known to be consumed.  A group's last wait of a tile showed that all slots up to 7 + n_pairs before the first
// of its next tile are; the parity needs 12 before.  From six pairs on the groups therefore take alternate pairs of every
// tile instead: each then owns three slots and waits for every use of them.
// One warp issues the MMAs, M 128 x N 32; four warps read the finished features and store them.  The gatherers wait for
// nothing but a free slot, so the loads, which bound the kernel (192 bytes per texel and pair through the L1 -> register
// port), never pause for a projection.
// Tensor memory: the ring [0, 432), two feature accumulators [448, 512).
//
// Every wait is bounded; when one runs out the CTA raises status[GNR_ST_WAIT_EXPIRED] and all its roles stop.
#include "gnr_gather.cuh"
#include "gnr_split.cuh"

namespace {

constexpr int GATHER_WARPS = 16, DRAIN_WARPS = 4;
constexpr int THREADS = (GATHER_WARPS + DRAIN_WARPS + 1) * 32;
constexpr int SLOTS = 6;
constexpr int F_COL = 448;

struct ProjectArgs {
  GnrCoords crd;
  const unsigned char* basis;  // [term][k group][32][8]
  float* feat_out;             // [n][FEAT_STRIDE]
  int32_t* status;
  uint32_t wait_limit;
  int debug_skip_commit;       // test hook: CTA 0 leaves out the commit of its first features
};

struct __align__(32) F8 {
  float2 v[4];
};
__device__ __forceinline__ F8 ldg8(const float* ptr) {
  F8 r;
  asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=f"(r.v[0].x), "=f"(r.v[0].y), "=f"(r.v[1].x), "=f"(r.v[1].y), "=f"(r.v[2].x), "=f"(r.v[2].y), "=f"(r.v[3].x), "=f"(r.v[3].y)
      : "l"(ptr));
  return r;
}

template <int MODE, int J, int NP>
__global__ void __launch_bounds__(THREADS, 1)
project_split_kernel(const __grid_constant__ GnrSampleParams p, const __grid_constant__ PlaneSet planes, const __grid_constant__ ProjectArgs a) {
  using T = Split<MODE>;
  constexpr int C = 16 * J;            // channels per pair
  constexpr int TERM_COLS = 8 * J;     // columns of one term of a slot
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t basis_bytes = (uint32_t)(planes.n * 2 * J * KGB_BYTES);  // one term
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + T::TW * basis_bytes);
  enum { FULL = 0, EMPTY = SLOTS, F_READY = 2 * SLOTS, F_FREE = F_READY + 2, WEIGHTS = F_FREE + 2, DRAIN, N_BARS };
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_bar + N_BARS);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  griddep_wait();
  const long long total = coords_total(a.crd);
  const long long n_tiles = (total + ROWS - 1) / ROWS;
  // a contiguous share of the list per CTA: neighbouring tiles read the same texels
  const long long per = (n_tiles + gridDim.x - 1) / gridDim.x;
  const long long t_beg = min(n_tiles, (long long)blockIdx.x * per);
  const int my_tiles = (int)(min(n_tiles, t_beg + per) - t_beg);
  if (my_tiles <= 0) return;  // (the whole CTA)
  const uint32_t bars = smem_u32(s_bar);
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  const int n_pairs = NP == 3 ? 3 : planes.n;

  if (warp == GATHER_WARPS + DRAIN_WARPS) {
    if (lane == 0) {
      for (int s = 0; s < SLOTS; ++s) {
        mbar_init(bar(FULL + s), GATHER_WARPS / 2);
        mbar_init(bar(EMPTY + s), 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(bar(F_READY + i), 1);
        mbar_init(bar(F_FREE + i), DRAIN_WARPS);
      }
      mbar_init(bar(WEIGHTS), 1);
      mbar_init(bar(DRAIN), 1);
      *s_abort = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    if (lane == 0) {
      mbar_expect_tx(bar(WEIGHTS), T::TW * basis_bytes);
      bulk_load(smem_u32(smem), a.basis, T::TW * basis_bytes, bar(WEIGHTS));
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);

  if (warp == GATHER_WARPS + DRAIN_WARPS) {
    // ---- MMAs, slots strictly in order -------------------------------------------------------------------------------
    constexpr uint32_t kIdesc = kIdescBasis | T::kFormat;
    bool ok = warp_wait(bar(WEIGHTS), 0, s_abort, a.status, a.wait_limit);
    const uint32_t wb = smem_u32(smem);
    int q = 0;
    for (int n = 0; n < my_tiles && ok; ++n) {
      const uint32_t f = tmem + F_COL + (uint32_t)(n & 1) * NB;
      auto products = [&](int i, int pi, uint32_t leader) {
        const uint32_t at = tmem + (uint32_t)((q + pi) % SLOTS) * (T::TA * TERM_COLS) + T::a(i) * TERM_COLS;
        const uint32_t b = wb + T::w(i) * basis_bytes + (uint32_t)pi * 2 * J * KGB_BYTES;
#pragma unroll
        for (int ks = 0; ks < J; ++ks)
          mma_f16_ts(f, at + ks * 8, make_desc(b + ks * 2 * KGB_BYTES, KGB_BYTES), kIdesc, (pi > 0 || i > 0 || ks > 0) ? 1u : 0u, leader);
      };
#pragma unroll 1
      for (int pi = 0; pi < n_pairs && ok; ++pi) {
        ok = warp_wait(bar(FULL + (q + pi) % SLOTS), (uint32_t)((q + pi) / SLOTS) & 1u, s_abort, a.status, a.wait_limit);
        if (ok && pi == 0 && n >= 2)  // the features of the tile two before must have been read
          ok = warp_wait(bar(F_FREE + (n & 1)), (uint32_t)((n >> 1) - 1) & 1u, s_abort, a.status, a.wait_limit);
        if (!ok) break;
        tc_fence_after();
        const uint32_t leader = elect_one();
#pragma unroll
        for (int i = 0; i + 1 < T::PRODUCTS; ++i) products(i, pi, leader);
        // more pairs than the ring holds beside the ones in work: their leading products cannot wait for the others
        if (n_pairs > SLOTS / 2) {
          products(T::PRODUCTS - 1, pi, leader);
          mma_commit(bar(EMPTY + (q + pi) % SLOTS), leader);
        }
      }
      if (!ok) break;
      const uint32_t leader = elect_one();
      if (n_pairs <= SLOTS / 2) {
#pragma unroll 1
        for (int pi = 0; pi < n_pairs; ++pi) {
          products(T::PRODUCTS - 1, pi, leader);
          mma_commit(bar(EMPTY + (q + pi) % SLOTS), leader);
        }
      }
      const bool skip = a.debug_skip_commit != 0 && blockIdx.x == 0 && n == 0;
      mma_commit(bar(F_READY + (n & 1)), skip ? 0u : leader);
      __syncwarp();
      q += n_pairs;
    }
    if (!ok) {
      // stop: wait (bounded, whatever limit the other waits have) until nothing of this CTA runs in the tensor pipe and
      // no copy of the weights still writes its shared memory
      mma_commit(bar(DRAIN), elect_one());
      __syncwarp();
      for (uint32_t it = 0; it < kWaitLimit && !mbar_try_wait(bar(DRAIN), 0); ++it) __nanosleep(64);
      for (uint32_t it = 0; it < kWaitLimit && !mbar_try_wait(bar(WEIGHTS), 0); ++it) __nanosleep(64);
    }
  } else if (warp >= GATHER_WARPS) {
    // ---- features: tensor memory -> global ------------------------------------------------------------------------------
    const int row = ((warp & 3) << 5) | lane;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    for (int n = 0; n < my_tiles; ++n) {
      if (!warp_wait(bar(F_READY + (n & 1)), (uint32_t)(n >> 1) & 1u, s_abort, a.status, a.wait_limit)) break;
      tc_fence_after();
      uint32_t v[32];
      tmem_ld32(tmem + F_COL + (uint32_t)(n & 1) * NB + lane_off, v);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(F_FREE + (n & 1)));
      const long long j = (t_beg + n) * ROWS + row;
      if (j < total) {
        float4* out = reinterpret_cast<float4*>(a.feat_out + (size_t)j * FEAT_STRIDE);
#pragma unroll
        for (int e = 0; e < FEAT_STRIDE / 4; ++e)
          out[e] = make_float4(__uint_as_float(v[4 * e]), __uint_as_float(v[4 * e + 1]), __uint_as_float(v[4 * e + 2]), __uint_as_float(v[4 * e + 3]));
      }
    }
  } else {
    // ---- gather -------------------------------------------------------------------------------------------------------------
    const int g = warp >> 3, wg = warp & 7, half = wg >> 2, row = ((wg & 3) << 5) | lane;
    const uint32_t lane_off = (uint32_t)((wg & 3) * 32) << 16;
    const bool by_pairs = n_pairs >= SLOTS;
    bool ok = true;
    for (int n = by_pairs ? 0 : g; n < my_tiles && ok; n += by_pairs ? 1 : 2) {
      const long long j = (t_beg + n) * ROWS + row;
      float x, y, z;
      sample_xyz(p, a.crd, j < total ? j : total - 1, x, y, z);  // (rows past the end repeat the last sample)
      Tap tx, ty, tz;
      if (NP == 3) {
        tx = make_tap(x, planes.p[0].fw, planes.p[0].W);
        ty = make_tap(y, planes.p[0].fh, planes.p[0].H);
        tz = make_tap(z, planes.p[0].fl, planes.p[0].L);
      }
#pragma unroll 1
      for (int pi = by_pairs ? (g + n * n_pairs) & 1 : 0; pi < n_pairs && ok; pi += by_pairs ? 2 : 1) {
        const GnrPlane& pl = planes.p[pi];
        Tap tu, tv, tl;
        if (NP == 3) {
          tu = pi == 2 ? ty : tx;
          tv = pi == 0 ? ty : tz;
          tl = pi == 0 ? tz : pi == 1 ? ty : tx;
        } else {
          tu = make_tap(pick(x, y, z, pl.mat0), pl.fw, pl.W);
          tv = make_tap(pick(x, y, z, pl.mat1), pl.fh, pl.H);
          tl = make_tap(pick(x, y, z, pl.vec), pl.fl, pl.L);
        }
        const float ax1 = tu.f1, ay1 = tv.f1, al1 = tl.f1;
        const float ax0 = 1.0f - ax1, ay0 = 1.0f - ay1, al0 = 1.0f - al1;
        const float w_nw = ax0 * ay0, w_ne = ax1 * ay0, w_sw = ax0 * ay1, w_se = ax1 * ay1;
        const uint32_t nw_t = (uint32_t)tv.i0 * (uint32_t)pl.W + (uint32_t)tu.i0;
        const float* nw_p = pl.plane + (size_t)nw_t * C + half * (C / 2);
        const float* sw_p = nw_p + (size_t)pl.W * C;
        const float* l_p = pl.line + (size_t)tl.i0 * C + half * (C / 2);
        const int q = n * n_pairs + pi, slot = q % SLOTS, use = q / SLOTS;
        const uint32_t at = tmem + lane_off + (uint32_t)slot * (T::TA * TERM_COLS) + (uint32_t)half * (TERM_COLS / 2);
#pragma unroll
        for (int h = 0; h < J; ++h) {  // eight channels per round
          const F8 nw = ldg8(nw_p + 8 * h), ne = ldg8(nw_p + C + 8 * h), sw = ldg8(sw_p + 8 * h), se = ldg8(sw_p + C + 8 * h);
          const F8 l0 = ldg8(l_p + 8 * h), l1 = ldg8(l_p + C + 8 * h);
          uint32_t t[T::TA][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float2 pv = __fmul2_rn(nw.v[e], make_float2(w_nw, w_nw));
            pv = __ffma2_rn(ne.v[e], make_float2(w_ne, w_ne), pv);
            pv = __ffma2_rn(sw.v[e], make_float2(w_sw, w_sw), pv);
            pv = __ffma2_rn(se.v[e], make_float2(w_se, w_se), pv);
            const float2 lv = __ffma2_rn(l1.v[e], make_float2(al1, al1), __fmul2_rn(l0.v[e], make_float2(al0, al0)));
            const float2 prod = __fmul2_rn(pv, lv);
            uint32_t terms[T::TA];
            T::split(prod.x, prod.y, terms);
#pragma unroll
            for (int i = 0; i < T::TA; ++i) t[i][e] = terms[i];
          }
          if (h == 0) {
            if (use > 0) ok = warp_wait(bar(EMPTY + slot), (uint32_t)(use - 1) & 1u, s_abort, a.status, a.wait_limit);
            if (!ok) break;
            tc_fence_after();
          }
#pragma unroll
          for (int i = 0; i < T::TA; ++i) tmem_st4(at + (uint32_t)(i * TERM_COLS + 4 * h), t[i]);
        }
        if (!ok) break;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(FULL + slot));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == GATHER_WARPS + DRAIN_WARPS) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

template <int MODE, int J, int NP>
int launch_variant(const GnrModel* m, const GnrSampleParams& p, const PlaneSet& set, const ProjectArgs& a, cudaStream_t st) {
  const size_t smem = (size_t)Split<MODE>::TW * set.n * 2 * J * KGB_BYTES + (2 * SLOTS + 6) * 8 + 16;
  cudaError_t e = cudaFuncSetAttribute(project_split_kernel<MODE, J, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int rc = gnr_launch(project_split_kernel<MODE, J, NP>, m->sm_count, THREADS, smem, st, a.crd.chained, p, set, a);
  if (rc) return rc;
  return (int)cudaGetLastError();
}

template <int MODE>
int launch_mode(const GnrModel* m, const GnrSampleParams& p, const PlaneSet& set, const ProjectArgs& a, cudaStream_t st) {
  const int J = set.p[0].C / 16;
  if (J == 3) return standard_vm3(set) ? launch_variant<MODE, 3, 3>(m, p, set, a, st) : launch_variant<MODE, 3, 0>(m, p, set, a, st);
  return J == 2 ? launch_variant<MODE, 2, 0>(m, p, set, a, st) : launch_variant<MODE, 1, 0>(m, p, set, a, st);
}

}  // namespace

// Mode 1 projects in two fp16 terms (one for the weights) where its products fit one operand buffer, as it always has;
// with more of them its features are fp32 ones from the CUDA cores.
int gnr_project_split_usable(const GnrModel* m) {
  return gnr_mlp_split_usable(m) && m->cfg.app_storage == 0 && m->app[0].C >= 16 && m->app[0].C <= 48 &&
         (m->cfg.mlp_mode == 0 || m->mlp.n_prod + 8 <= MAX_K0);
}

int launch_project_split(const GnrModel* m, const GnrSampleParams& p, const GnrCoords& c, int feat_stride, float* feat,
                         int32_t* status, cudaStream_t st) {
  if (!m->mlp.split_basis || feat_stride != FEAT_STRIDE) {
    gnr_set_error("split projection: weights were not prepared, or feature stride %d is not %d", feat_stride, FEAT_STRIDE);
    return -1;
  }
  ProjectArgs a;
  a.crd = c;
  a.basis = (const unsigned char*)m->mlp.split_basis;
  a.feat_out = feat;
  a.status = status;
  a.wait_limit = m->debug_wait_limit > 0 ? (uint32_t)m->debug_wait_limit : kWaitLimit;
  a.debug_skip_commit = m->debug_expire_wait == GNR_EXPIRE_ANY || m->debug_expire_wait == GNR_EXPIRE_PROJECTION;
  const PlaneSet set = make_set(m->app, m->cfg.n_pairs);
  return m->cfg.mlp_mode == 0 ? launch_mode<0>(m, p, set, a, st) : launch_mode<1>(m, p, set, a, st);
}
