// Appearance MLP (150 -> 128 -> 128 -> 3) on the tensor cores with every operand carried as a sum of 16-bit terms.
//
// MLPRender_Fea.forward (app/models/mlp_render_fea.py:44-68) with positional_encoding
// (app/tools/utils.py:42-48): input = [feat, view, sin(feat 2^f), cos(feat 2^f), sin(view 2^f), cos(view 2^f)].
//
// mlp_mode 0: the fp32 network, operands as exact sums of three bf16 terms; mlp_mode 1: activations as fp16 hi + lo (see
// gnr_split.cuh).  Biases, ReLU, the encodings and layer 3 are fp32 on the CUDA cores.
//
// Work split: one persistent CTA per SM, tiles of 128 samples (row = lane of tensor memory), three roles.
//   * eight warps ENCODE (two threads per row): layer 1's input travels in chunks of 32 columns (two K steps) through a
//     ring of slots in tensor memory.  The K order of layer 1 is permuted so that each K step holds three values u with
//     their sin u, sin 2u, cos u, cos 2u (and one zero): a thread encodes three values, splits 16 numbers, and stores 8
//     columns per term.  A slot is free when the MMAs of its chunk have completed (tcgen05.commit).
//   * eight warps FINISH: relu(D1 + b1) becomes layer 2's input IN PLACE, terms h and m over the columns of D1 just read
//     (term l beside it), so that the ring belongs to layer 1 alone and the next tile is encoded while this one goes
//     through layer 2; then layer 3 from D2.
//   * one warp issues every MMA.
// Leading products are issued last, after the small ones of the layer: the sums in tensor memory do not round to nearest,
// and this way few steps happen at full size (with three terms the ring holds four of the five chunks, so the fifth's
// small products come after the leading ones of the first).  Error against fp64 on 119,185 samples: rms 2.3e-8; 2.6e-8
// with all products chunk by chunk; 2.35e-8 with fp32 arithmetic on the CUDA cores.
// What bounds it: the tensor pipe (70 % active: 108 MMAs of 78 cycles per tile with three terms, 8400 of 11,300 cycles),
// then the chain D1 -> first chunk of layer 2.  752,149 samples: 237 us; 1,900 in fp32 on the CUDA cores; 327 with all
// sixteen warps encoding and converting the same tile, 312 with two groups of warps on alternate tiles (in both, layer
// 2's input took ring slots, so a tile could not be encoded while the one before was in the tensor pipe).
// Tensor memory: D1 (layer 1 result, then terms h and m of layer 2's input) [0, 128), D2 [128, 256), term l [256, 320),
// the ring [320, 512).  Shared memory: the weight images (216 KB with three terms), biases, layer-3 weights.
//
// Every wait is bounded; when one runs out the CTA raises status[GNR_ST_WAIT_EXPIRED] and all its roles stop.
#include "gnr_split.cuh"

namespace {

constexpr int ROLE_WARPS = 8;              // warps that encode, and warps that finish (two threads per row)
constexpr int MMA_WARP = 2 * ROLE_WARPS;
constexpr int THREADS = (2 * ROLE_WARPS + 1) * 32;
constexpr int L1_CHUNKS = 5, L2_CHUNKS = 4;
constexpr int CHUNK_COLS = 16;             // tensor-memory columns of one term of a chunk (32 values)
constexpr int L_COL = 256, RING_COL = 320;
constexpr int MAX_BARS = 24;
constexpr int W1S_BYTES = 160 * HID * 2, W2S_BYTES = HID * HID * 2;  // one term of a weight image

struct SplitArgs {
  GnrCoords crd;
  const float* feat;             // [n][FEAT_STRIDE]
  const unsigned char* w_image;  // [term][W1 image, permuted K][...], then [term][W2 image]
  const float* w3;
  const float* b1;
  const float* b2;
  const float* b3;
  float* rgb_out;
  int32_t* status;
  int kbits;
  uint32_t wait_limit;
  int debug_skip_commit;         // test hook: CTA 0 leaves out the commit of its first layer-1 result
};

template <int MODE>
__global__ void __launch_bounds__(THREADS, 1) mlp_split_kernel(const __grid_constant__ SplitArgs a) {
  using T = Split<MODE>;
  constexpr int SLOT_COLS = T::TA * CHUNK_COLS, SLOTS = (512 - RING_COL) / SLOT_COLS;  // 4 with three terms, 6 with two
  constexpr int AHEAD = SLOTS < L1_CHUNKS ? SLOTS : L1_CHUNKS;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* s_w1 = smem;                                  // [TW][W1S_BYTES]
  unsigned char* s_w2 = s_w1 + T::TW * W1S_BYTES;              // [TW][W2S_BYTES]
  float* s_w3 = reinterpret_cast<float*>(s_w2 + T::TW * W2S_BYTES);  // [3][HID]
  float* s_b1 = s_w3 + 3 * HID;
  float* s_b2 = s_b1 + HID;
  float* s_b3 = s_b2 + HID;                                    // [4]
  float* s_part = s_b3 + 4;                                    // [128][3] layer-3 sums of the second half of a row
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(s_part + ROWS * 3);
  enum { FULL = 0, EMPTY = SLOTS, A2_FULL = 2 * SLOTS, D1_READY = A2_FULL + L2_CHUNKS, D2_READY, D2_FREE, WEIGHTS, DRAIN, PART, N_BARS };
  static_assert(N_BARS <= MAX_BARS, "barriers");
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(s_bar + N_BARS);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const uint32_t bars = smem_u32(s_bar);
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  auto wait = [&](int i, uint32_t parity) { return warp_wait(bar(i), parity & 1u, s_abort, a.status, a.wait_limit); };

  // ---- set-up: barriers, tensor memory; the weight images come in by bulk copies while the first tile is encoded ----
  constexpr uint32_t kImage = T::TW * (W1S_BYTES + W2S_BYTES);
  if (warp == MMA_WARP) {
    if (lane == 0) {
      for (int s = 0; s < SLOTS; ++s) {
        mbar_init(bar(FULL + s), ROLE_WARPS);
        mbar_init(bar(EMPTY + s), 1);
      }
      for (int c = 0; c < L2_CHUNKS; ++c) mbar_init(bar(A2_FULL + c), ROLE_WARPS);
      mbar_init(bar(D1_READY), 1);
      mbar_init(bar(D2_READY), 1);
      mbar_init(bar(D2_FREE), ROLE_WARPS);
      mbar_init(bar(WEIGHTS), 1);
      mbar_init(bar(DRAIN), 1);
      mbar_init(bar(PART), ROLE_WARPS / 2);
      *s_abort = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (lane == 0) {
      mbar_expect_tx(bar(WEIGHTS), kImage);
      for (uint32_t at = 0; at < kImage; at += 16384u)
        bulk_load(smem_u32(smem) + at, a.w_image + at, min(16384u, kImage - at), bar(WEIGHTS));
    }
    __syncwarp();
  } else {
    for (int i = tid; i < 3 * HID; i += MMA_WARP * 32) s_w3[i] = a.w3[i];
    if (tid < HID) {
      s_b1[tid] = a.b1[tid];
      s_b2[tid] = a.b2[tid];
    }
    if (tid < 4) s_b3[tid] = a.b3[tid];
  }
  griddep_wait();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  const long long total = min(a.crd.total_ptr ? (long long)*a.crd.total_ptr : a.crd.total_direct, a.crd.capacity);
  const long long n_tiles = (total + ROWS - 1) / ROWS;
  const int my_tiles = (int)max(0LL, (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *s_tmem, 0);
  const uint32_t d1 = tmem, d2 = tmem + HID, l2_low = tmem + L_COL, ring = tmem + RING_COL;

  if (warp == MMA_WARP) {
    // ---- MMAs ------------------------------------------------------------------------------------------------------------
    // (WAR: layer 1 of the next tile overwrites D1, whose columns hold layer 2's operand; MMAs of one thread run in order)
    constexpr uint32_t kIdesc = kIdescHid | T::kFormat;
    bool ok = wait(WEIGHTS, 0);
    const uint32_t w1 = smem_u32(s_w1), w2 = smem_u32(s_w2);
    int q = 0;  // chunks of layer 1 taken so far
    for (int n = 0; n < my_tiles && ok; ++n) {
      // layer 1
      auto products1 = [&](int i, int c, uint32_t leader) {
        const uint32_t at = ring + (uint32_t)((q + c) % SLOTS) * SLOT_COLS + T::a(i) * CHUNK_COLS;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks)
          mma_f16_ts(d1, at + ks * 8, make_desc(w1 + T::w(i) * W1S_BYTES + (uint32_t)(4 * c + 2 * ks) * KG_BYTES, KG_BYTES), kIdesc,
                     (c > 0 || i > 0 || ks > 0) ? 1u : 0u, leader);
      };
      int led = 0;  // chunks whose leading products have been issued
#pragma unroll 1
      for (int c = 0; c < L1_CHUNKS && ok; ++c) {
        ok = wait(FULL + (q + c) % SLOTS, (uint32_t)((q + c) / SLOTS));
        if (!ok) break;
        tc_fence_after();
        const uint32_t leader = elect_one();
#pragma unroll
        for (int i = 0; i + 1 < T::PRODUCTS; ++i) products1(i, c, leader);
        if (c + 1 >= AHEAD) {
          // all chunks are in: the leading products of the rest; a slot short: those of the first chunk, whose slot the
          // last one waits for
          const int upto = c + 1 == L1_CHUNKS ? L1_CHUNKS : L1_CHUNKS - AHEAD;
#pragma unroll 1
          for (; led < upto; ++led) {
            products1(T::PRODUCTS - 1, led, leader);
            mma_commit(bar(EMPTY + (q + led) % SLOTS), leader);
          }
        }
      }
      if (!ok) break;
      const bool skip = a.debug_skip_commit != 0 && blockIdx.x == 0 && n == 0;
      mma_commit(bar(D1_READY), skip ? 0u : elect_one());
      __syncwarp();
      q += L1_CHUNKS;
      // layer 2: chunk c = hidden units 16 c .. 16 c + 15 of either half (K steps c and 4 + c)
      auto products2 = [&](int i, int c, uint32_t leader) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t at = T::a(i) == 2 ? l2_low + 32 * h + 8 * c : d1 + 64 * h + 32 * T::a(i) + 8 * c;
          mma_f16_ts(d2, at, make_desc(w2 + T::w(i) * W2S_BYTES + (uint32_t)(8 * h + 2 * c) * KG_BYTES, KG_BYTES), kIdesc,
                     (c > 0 || i > 0 || h > 0) ? 1u : 0u, leader);
        }
      };
      if (n > 0) ok = wait(D2_FREE, (uint32_t)(n - 1));  // layer 2 of the tile before has been read out
#pragma unroll 1
      for (int c = 0; c < L2_CHUNKS && ok; ++c) {
        ok = wait(A2_FULL + c, (uint32_t)n);
        if (!ok) break;
        tc_fence_after();
        const uint32_t leader = elect_one();
#pragma unroll
        for (int i = 0; i + 1 < T::PRODUCTS; ++i) products2(i, c, leader);
      }
      if (!ok) break;
      const uint32_t leader = elect_one();
#pragma unroll
      for (int c = 0; c < L2_CHUNKS; ++c) products2(T::PRODUCTS - 1, c, leader);
      mma_commit(bar(D2_READY), leader);
      __syncwarp();
    }
    if (!ok) {
      // stop: wait (bounded, whatever limit the other waits have) until nothing of this CTA runs in the tensor pipe and
      // no copy of the weights still writes its shared memory
      mma_commit(bar(DRAIN), elect_one());
      __syncwarp();
      for (uint32_t it = 0; it < kWaitLimit && !mbar_try_wait(bar(DRAIN), 0); ++it) __nanosleep(64);
      for (uint32_t it = 0; it < kWaitLimit && !mbar_try_wait(bar(WEIGHTS), 0); ++it) __nanosleep(64);
    }
  } else {
    const int wg = warp & (ROLE_WARPS - 1);
    const int half = wg >> 2, row = ((wg & 3) << 5) | lane;
    const uint32_t lane_off = (uint32_t)((wg & 3) * 32) << 16;
    auto tile_row = [&](int n) { return ((long long)blockIdx.x + (long long)n * gridDim.x) * ROWS + row; };
    // 16 numbers -> T::TA terms of eight packed columns
    auto split16 = [&](const float (&x)[16], uint32_t (&t)[T::TA][8]) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        uint32_t terms[T::TA];
        T::split(x[2 * e], x[2 * e + 1], terms);
#pragma unroll
        for (int i = 0; i < T::TA; ++i) t[i][e] = terms[i];
      }
    };
    bool ok = true;
    if (my_tiles == 0) {
      // (only the copies of the weights to see out, by the MMA warp)
    } else if (warp < ROLE_WARPS) {
      // ---- encode --------------------------------------------------------------------------------------------------------
      // this thread's three values of chunk c: 6 c + 3 half .. of the features; the last three of half 1 are the view direction
      const uint32_t ring_half = ring + lane_off + (uint32_t)(half * 8);  // this thread's 8 of a term's 16 columns
      const float *fr, *last;
      auto row_sources = [&](int n) {
        const long long j = tile_row(n), js = j < total ? j : total - 1;
        fr = a.feat + (size_t)js * FEAT_STRIDE + 3 * half;
        last = fr + 6 * (L1_CHUNKS - 1);
        if (half == 1) {
          if (a.crd.view_direct) {
            last = a.crd.view_direct + (size_t)js * a.crd.point_stride;
          } else {
            const uint32_t ray = __ldg(a.crd.ids + (a.crd.index ? (long long)__ldg(a.crd.index + js) : js)) >> a.kbits;
            last = a.crd.rays + (size_t)ray * 6 + 3;
          }
        }
      };
      auto load = [&](int c, float (&u)[3]) {
        const float* src = c + 1 < L1_CHUNKS ? fr + 6 * c : last;
#pragma unroll
        for (int i = 0; i < 3; ++i) u[i] = __ldg(src + i);
      };
      float u[3], ahead[3];
      row_sources(0);
      load(0, u);
      const int chunks = my_tiles * L1_CHUNKS;
      int c = 0;  // chunk in its tile
      // (not unrolled: the encoding is long, and unrolled it does not fit the instruction cache)
#pragma unroll 1
      for (int q = 0; q < chunks && ok; ++q) {
        if (++c == L1_CHUNKS) {
          c = 0;
          if (q + 1 < chunks) row_sources(q / L1_CHUNKS + 1);
        }
        load(c, ahead);  // the values of the next chunk (behind the last one: the same row again)
        float x[16];
        T::encode(u, x);
        uint32_t t[T::TA][8];
        split16(x, t);
        const int slot = q % SLOTS;
        if (q >= SLOTS) ok = wait(EMPTY + slot, (uint32_t)(q / SLOTS - 1));
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int i = 0; i < T::TA; ++i) tmem_st8(ring_half + (uint32_t)(slot * SLOT_COLS + i * CHUNK_COLS), t[i]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(FULL + slot));
#pragma unroll
        for (int i = 0; i < 3; ++i) u[i] = ahead[i];
      }
    } else {
      // ---- finish ----------------------------------------------------------------------------------------------------------
      const uint32_t d1_half = d1 + lane_off + 64u * (uint32_t)half, low_half = l2_low + lane_off + 32u * (uint32_t)half;
#pragma unroll 1
      for (int n = 0; n < my_tiles; ++n) {
        // layer 2's input: relu(D1 + b1), 16 of this half's 64 units at a time; the upper 32 columns are read before term m
        // overwrites them
        if (!(ok = wait(D1_READY, (uint32_t)n))) break;
        tc_fence_after();
        uint32_t upper[32], v[16];
        tmem_ld16(d1_half, v);
        tmem_ld32(d1_half + 32, upper);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < L2_CHUNKS; ++c) {
          float x[16];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 b = *reinterpret_cast<const float4*>(s_b1 + 64 * half + 16 * c + 4 * e);
            const float bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t raw = c < 2 ? v[4 * e + i] : upper[16 * (c - 2) + 4 * e + i];
              x[4 * e + i] = fmaxf(__uint_as_float(raw) + bb[i], 0.0f);
            }
          }
          uint32_t t[T::TA][8];
          split16(x, t);
          if (c == 0) {  // the next 16 columns, before the first 8 are overwritten
            tmem_ld16(d1_half + 16, v);
            tmem_ld_wait();
          }
          tmem_st8(d1_half + 8 * c, t[0]);
          tmem_st8(d1_half + 32 + 8 * c, t[1]);
          if constexpr (T::TA == 3) tmem_st8(low_half + 8 * c, t[2]);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(A2_FULL + c));
        }
        // layer 3: rgb = sigmoid(W3 relu(D2 + b2) + b3), fp32; half h sums columns 64 h ..
        if (!(ok = wait(D2_READY, (uint32_t)n))) break;
        tc_fence_after();
        float2 p0 = make_float2(0.0f, 0.0f), p1 = p0, p2 = p0;
#pragma unroll
        for (int cb = 0; cb < 2; ++cb) {
          const int col = 64 * half + 32 * cb;
          tmem_ld32(d2 + lane_off + col, upper);
          tmem_ld_wait();
          if (cb == 1) {  // the accumulator can be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(D2_FREE));
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float4 b = *reinterpret_cast<const float4*>(s_b2 + col + 4 * e);
            const float2 xa = make_float2(fmaxf(__uint_as_float(upper[4 * e + 0]) + b.x, 0.0f), fmaxf(__uint_as_float(upper[4 * e + 1]) + b.y, 0.0f));
            const float2 xb = make_float2(fmaxf(__uint_as_float(upper[4 * e + 2]) + b.z, 0.0f), fmaxf(__uint_as_float(upper[4 * e + 3]) + b.w, 0.0f));
            const float4 wr = *reinterpret_cast<const float4*>(s_w3 + col + 4 * e);
            const float4 wg4 = *reinterpret_cast<const float4*>(s_w3 + HID + col + 4 * e);
            const float4 wb4 = *reinterpret_cast<const float4*>(s_w3 + 2 * HID + col + 4 * e);
            p0 = __ffma2_rn(xb, make_float2(wr.z, wr.w), __ffma2_rn(xa, make_float2(wr.x, wr.y), p0));
            p1 = __ffma2_rn(xb, make_float2(wg4.z, wg4.w), __ffma2_rn(xa, make_float2(wg4.x, wg4.y), p1));
            p2 = __ffma2_rn(xb, make_float2(wb4.z, wb4.w), __ffma2_rn(xa, make_float2(wb4.x, wb4.y), p2));
          }
        }
        float* part = s_part + row * 3;
        // (half 1 cannot overtake: its next sums follow MMAs that need half 0's next chunks, stored after the reads here)
        if (half == 1) {
          part[0] = p0.x + p0.y;
          part[1] = p1.x + p1.y;
          part[2] = p2.x + p2.y;
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(PART));
          continue;
        }
        if (!(ok = wait(PART, (uint32_t)n))) break;
        const long long j = tile_row(n);
        if (j < total) {
          float* out = a.rgb_out + (size_t)j * 3;
          out[0] = 1.0f / (1.0f + expf(-((p0.x + p0.y) + part[0] + s_b3[0])));
          out[1] = 1.0f / (1.0f + expf(-((p1.x + p1.y) + part[1] + s_b3[1])));
          out[2] = 1.0f / (1.0f + expf(-((p2.x + p2.y) + part[2] + s_b3[2])));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// W [n_out][k_real] fp32 -> [term][k group][n_rows][8] 16-bit terms; rows past n_out are zero.  KIND: where position k of
// the operand comes from: 0 = column k, 1 = the K order of layer 1, 2 = products of pairs padded from c to cp channels.
template <int MODE, int KIND>
__global__ void pack_split_image_kernel(const float* __restrict__ w, uint16_t* __restrict__ img, int n_out, int n_rows, int k_real,
                                        int k_groups, int c, int cp) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // one thread per (k group, n)
  if (i >= k_groups * n_rows) return;
  const int kg = i / n_rows, n = i - kg * n_rows;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int k = kg * 8 + e;
    int col = k;
    if (KIND == 1) {
      // K step s = k / 16 holds the values 3 s .. 3 s + 2 (features, then view), each as u, sin u, sin 2u, cos u, cos 2u
      const int r = k & 15, v = 3 * (k >> 4) + r / 5, what = r % 5;
      const bool view = v >= APP;
      const int base_s = APP + 3, base_vs = base_s + 4 * APP;
      const int sin0 = view ? base_vs + 2 * (v - APP) : base_s + 2 * v;
      const int cos0 = sin0 + (view ? 6 : 2 * APP);
      col = r == 15 ? -1 : what == 0 ? v : what <= 2 ? sin0 + what - 1 : cos0 + what - 3;
    } else if (KIND == 2) {
      const int pair = k / cp, ch = k - pair * cp;
      col = ch < c ? pair * c + ch : -1;
    }
    float x = (n < n_out && col >= 0 && col < k_real) ? w[(size_t)n * k_real + col] : 0.0f;
#pragma unroll
    for (int t = 0; t < Split<MODE>::TW; ++t) img[((size_t)t * k_groups * n_rows + i) * 8 + e] = Split<MODE>::term(x);
  }
}

// [layer 1: TW terms][layer 2: TW terms][basis: TW terms], the basis only where the products fit one operand
template <int MODE>
int prepare_images(GnrModel* m, const float* basis_w, const float* w1, const float* w2, cudaStream_t st) {
  constexpr int TW = Split<MODE>::TW;
  const size_t net = (size_t)TW * (W1S_BYTES + W2S_BYTES);
  const int cp = (m->cfg.n_app + 15) / 16 * 16, kgb = m->cfg.n_pairs * cp / 8;
  if (m->mlp.split_image == nullptr) GNR_CUDA_OK(cudaMalloc(&m->mlp.split_image, net + (size_t)TW * kgb * KGB_BYTES));
  unsigned char* img = (unsigned char*)m->mlp.split_image;
  pack_split_image_kernel<MODE, 1><<<(20 * HID + 255) / 256, 256, 0, st>>>(w1, (uint16_t*)img, HID, HID, IN_DIM, 20, 0, 0);
  pack_split_image_kernel<MODE, 0><<<(16 * HID + 255) / 256, 256, 0, st>>>(w2, (uint16_t*)(img + (size_t)TW * W1S_BYTES), HID, HID, HID,
                                                                          16, 0, 0);
  m->mlp.split_basis = img + net;
  pack_split_image_kernel<MODE, 2><<<(kgb * NB + 255) / 256, 256, 0, st>>>(basis_w, (uint16_t*)m->mlp.split_basis, m->cfg.app_dim, NB,
                                                                          m->cfg.n_pairs * m->cfg.n_app, kgb, m->cfg.n_app, cp);
  GNR_CUDA_OK(cudaGetLastError());
  return 0;
}

template <int MODE>
int launch_mode(const GnrModel* m, const SplitArgs& a, cudaStream_t st) {
  constexpr size_t smem = (size_t)Split<MODE>::TW * (W1S_BYTES + W2S_BYTES) + (3 * HID + 2 * HID + 4 + ROWS * 3) * sizeof(float) +
                          MAX_BARS * 8 + 16;
  static_assert(smem <= 227 * 1024, "the weights of the split network must fit shared memory");
  cudaError_t e = cudaFuncSetAttribute(mlp_split_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int rc = gnr_launch(mlp_split_kernel<MODE>, m->sm_count, THREADS, smem, st, a.crd.chained, a);
  if (rc) return rc;
  return (int)cudaGetLastError();
}

}  // namespace

int gnr_mlp_split_usable(const GnrModel* m) {
  const GnrConfig& c = m->cfg;
  return c.mlp_mode <= 1 && c.app_dim == APP && c.fea_pe == FPE && c.view_pe == VPE && c.hidden == HID;
}

int gnr_mlp_split_prepare(GnrModel* m, const float* basis_w, const float* w1, const float* w2, cudaStream_t st) {
  return m->cfg.mlp_mode == 0 ? prepare_images<0>(m, basis_w, w1, w2, st) : prepare_images<1>(m, basis_w, w1, w2, st);
}

int launch_mlp_split(const GnrModel* m, const GnrSampleParams& p, const GnrCoords& c, int feat_stride, const float* feat,
                     float* rgb, int32_t* status, cudaStream_t st) {
  if (!m->mlp.split_image || feat_stride != FEAT_STRIDE) {
    gnr_set_error("split network: weights were not prepared, or feature stride %d is not %d", feat_stride, FEAT_STRIDE);
    return -1;
  }
  SplitArgs a;
  a.crd = c;
  a.feat = feat;
  a.w_image = (const unsigned char*)m->mlp.split_image;
  a.w3 = m->mlp.w3;
  a.b1 = m->mlp.b1;
  a.b2 = m->mlp.b2;
  a.b3 = m->mlp.b3;
  a.rgb_out = rgb;
  a.status = status;
  a.kbits = p.kbits;
  a.wait_limit = m->debug_wait_limit > 0 ? (uint32_t)m->debug_wait_limit : kWaitLimit;
  a.debug_skip_commit = m->debug_expire_wait == GNR_EXPIRE_ANY || m->debug_expire_wait == GNR_EXPIRE_NETWORK;
  return m->cfg.mlp_mode == 0 ? launch_mode<0>(m, a, st) : launch_mode<1>(m, a, st);
}
