// The W4A16 GEMM for batches of up to 8 rows, and 16 where latency decides: a stream of packed weights through CTAs of
// HALF an SM, multiplied with mma.sync straight from registers.
//
// What bounds these problems is not HBM alone: a layer of a few megabytes is over in the time that a CTA takes to start,
// and a whole-SM CTA of the tcgen05 kernel (w4a16_kernel_decode.cuh) starts only when the previous launch has left its SM:
// barriers, tensor-memory allocation, first bytes, then nibbles -> registers -> tensor memory -> MMA -> tensor memory ->
// registers, four hand-offs between warps.  Here a packed word goes from shared memory to the registers of the warp
// that multiplies it: the word is laid out as the A fragment of mma.m16n8k16 (marlin_cute_trait.h:8-39,644-686; weight
// columns are the 16 rows, 8 batch rows the n), so there is one hand-off (TMA -> warp) and no tensor memory.  Two CTAs share
// an SM, and under programmatic dependent launch the CTAs of the next launch of the stream move in, fill their rings with
// weights and wait for the activations only.  At 8 rows the MMAs take a third of the HBM time of the weights; at 16 two thirds
// (8 clocks per m16n8k16 and sub-partition), where the tcgen05 kernel is the faster one.
//
// us per launch in a chain, tcgen05 kernel -> this one (m = 1): see the rule in dispatch_tc.
#pragma once
#include "w4a16_kernel.cuh"

namespace w4a16 {

// MT: batch tiles of 8 rows (the n of mma.m16n8k16).  KS: k per stage; 128 for k an odd multiple of 128 and where the
// activations make a stage large.
template <int MT, int KS_>
struct SkinnyConfig {
  static_assert(MT == 1 || (MT == 2 && KS_ == 128), "8 or 16 batch rows");
  static_assert(KS_ == 256 || KS_ == 128, "k per stage");
  static constexpr int ROWS = 8 * MT;
  static constexpr int KS = KS_;
  static constexpr int GROUPS = KS / 128;
  // Consumer warps: 2 column blocks of 64 x 4 k-lanes, two on each of the SM's sub-partitions (with six of them and a producer,
  // 4 / 4 / 2 / 2 of the two CTAs' twelve, 16 x 57344 x 8192 took 70 us).  A ninth warp leaves a thread 96 registers; the
  // accumulators of 16 rows need 128, so there the consumers request the loads themselves.
  static constexpr int LANES = 4;
  static constexpr int NW = 2 * LANES;
  static constexpr bool PRODUCER = MT == 1;
  static constexpr int THREADS = (NW + (PRODUCER ? 1 : 0)) * 32;
  static constexpr int W_BYTES = KS * TILE_N / 2;            // [KS/16][256] words, as they lie in B
  static constexpr int A_BYTES = ROWS * KS * 2;              // [KS/64][ROWS][128 B], 128-byte swizzle
  static constexpr int S_BYTES = GROUPS * TILE_N * 2;
  static constexpr int STAGE_BYTES = W_BYTES + A_BYTES + S_BYTES;
  static constexpr int RED_LD = TILE_N + 4;                  // fp32 pitch of the reduction buffer
  static constexpr int RED_LANE = ROWS * RED_LD;             // cells of one k-lane
  // The lanes' sums lie side by side: in a buffer of their own at 8 rows; over the ring in the cluster form (its one tile has
  // been consumed by then), which has the other ranks' partial rows in that buffer; the stream-K form of 16 rows
  // has room for one lane and adds the others in turn.
  static constexpr int SK_LANES = MT == 1 ? LANES : 1;
  static constexpr int X_BYTES = SK_LANES * RED_LANE * 4;
  static constexpr int STAGES_RAW = (113 * 1024 - X_BYTES - 256 - 1024) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_RAW * KS > 1024 ? 1024 / KS : STAGES_RAW;
  static_assert(STAGES >= 3, "ring too shallow");
  static_assert(LANES * RED_LANE * 4 <= STAGES * (W_BYTES + A_BYTES), "the lanes' sums fit the ring");
  static_assert(ROWS * TILE_N * 4 <= X_BYTES, "the partial rows fit the reduction buffer");
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + X_BYTES + 256 /*barriers*/ + 1024 /*align slack*/;
  static_assert(SMEM_BYTES <= 113 * 1024, "two CTAs per SM");
};

struct SkinnyBars {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t slab;     // the other ranks' rows have arrived
  int abort;
};
static_assert(sizeof(SkinnyBars) <= 256, "barrier block");

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, bool zero) {
  if (zero) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void lds128(uint32_t (&v)[4], uint32_t addr) {
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(addr) : "memory");
}
// Four neighbouring cells of a partial-tile slot: each cell is its own flag (idle or written), so the vector access need
// not be atomic as a whole.
__device__ __forceinline__ void st_slot4(uint32_t *p, float4 v) {
  uint32_t x[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
#pragma unroll
  for (int e = 0; e < 4; ++e) x[e] = x[e] == PARTIAL_IDLE ? 0x7fffffffu : x[e];
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]) : "memory");
}
// Adds the cells that `count` other CTAs left at p, p + stride, ... in that order, and puts the idle pattern back.
__device__ __forceinline__ bool fold_slots4(float4 &v, uint32_t *p, int stride, int count, volatile int *abort, uint64_t wait_ns) {
  constexpr int FLY = 4;   // slices in flight
  const uint64_t t0 = sm100::globaltimer_ns();
  for (int j = 0; j < count; j += FLY) {
    uint32_t x[FLY][4];
    for (uint32_t spin = 0;; ++spin) {
      bool up = true;
#pragma unroll
      for (int f = 0; f < FLY; ++f)
        asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(x[f][0]), "=r"(x[f][1]), "=r"(x[f][2]), "=r"(x[f][3])
                     : "l"(p + (size_t)min(j + f, count - 1) * stride)
                     : "memory");
#pragma unroll
      for (int f = 0; f < FLY; ++f)
#pragma unroll
        for (int e = 0; e < 4; ++e) up &= x[f][e] != PARTIAL_IDLE;
      if (__all_sync(0xffffffffu, up)) break;
      if ((spin & 0xf) == 0xf && __any_sync(0xffffffffu, *abort || sm100::globaltimer_ns() - t0 > wait_ns)) return false;
    }
#pragma unroll
    for (int f = 0; f < FLY; ++f)
      if (j + f < count) {
        v.x += __uint_as_float(x[f][0]), v.y += __uint_as_float(x[f][1]), v.z += __uint_as_float(x[f][2]), v.w += __uint_as_float(x[f][3]);
        asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %1, %1, %1};" ::"l"(p + (size_t)(j + f) * stride), "r"(PARTIAL_IDLE) : "memory");
      }
  }
  return true;
}

// Work: 128-column tiles x stages.  Cluster form (cl > 1): one cluster of cl CTAs per tile, its k-range cut cl ways; rank r
// finishes rows r, r + cl, ..., the ranks send one another their partial rows through distributed shared memory.  Stream-K
// form (cl == 1): equal contiguous ranges, two CTAs make a worker.  CTA c (blocks counted backwards) finishes the tile whose
// first stage it holds and adds what CTAs c + 1, c + 2, ... leave in the scratch; those are LOWER block indices, so
// whatever a CTA waits for was dispatched before it.
template <int MT, int KS_, bool GROUPED>
__global__ void __launch_bounds__(SkinnyConfig<MT, KS_>::THREADS, 2)
w4a16_skinny_kernel(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmA,
                    const __grid_constant__ CUtensorMap tmS, const Params p, const int cl) {
  using Cfg = SkinnyConfig<MT, KS_>;
  using namespace sm100;
  constexpr int S = Cfg::STAGES, NW = Cfg::NW, GROUPS = Cfg::GROUPS, LANES = Cfg::LANES;
  constexpr uint32_t STAGE_TX = Cfg::W_BYTES + Cfg::A_BYTES + (GROUPED ? Cfg::S_BYTES : 0);

  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sW = smem;
  uint8_t *sA = sW + S * Cfg::W_BYTES;
  uint8_t *sS = sA + S * Cfg::A_BYTES;
  float *xbuf = reinterpret_cast<float *>(sS + S * Cfg::S_BYTES);
  SkinnyBars *bars = reinterpret_cast<SkinnyBars *>(reinterpret_cast<uint8_t *>(xbuf) + Cfg::X_BYTES);
  volatile int *abort = &bars->abort;
  float *red = cl > 1 ? reinterpret_cast<float *>(sW) : xbuf;
  float *slab = xbuf;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int tile, kk, total, rank = 0, cta = 0;
  if (cl > 1) {
    tile = blockIdx.x / cl;               // a cluster is cl consecutive blocks
    rank = blockIdx.x - tile * cl;
    kk = p.k_iters * rank / cl;
    total = p.k_iters * (rank + 1) / cl - kk;
  } else {
    cta = (int)(gridDim.x - 1 - blockIdx.x);
    const int it0 = cta * p.iters_per_cta;
    total = min(p.total_iters - it0, p.iters_per_cta);
    tile = it0 / p.k_iters;
    kk = it0 - tile * p.k_iters;
  }

  auto load_weights = [&](int st, int t, int k) {   // packed weights and scales: parameters
    const uint32_t full = smem_u32(&bars->full[st]);
    mbar_expect_tx(full, STAGE_TX);
    tma_load_2d(smem_u32(sW) + st * Cfg::W_BYTES, &tmB, t * 2 * TILE_N, k * (Cfg::KS / 16), full);
    if (GROUPED) tma_load_2d(smem_u32(sS) + st * Cfg::S_BYTES, &tmS, t * TILE_N, k * GROUPS, full);
  };
  auto load_acts = [&](int st, int k) { tma_load_3d(smem_u32(sA) + st * Cfg::A_BYTES, &tmA, 0, 0, k * (Cfg::KS / 64), smem_u32(&bars->full[st])); };

  // ---- prologue: barriers, then the first ring-full of weights
  const int first = min(S, total);
  if (warp == (Cfg::PRODUCER ? NW : 0)) {
    if (lane < S) {
      mbar_init(smem_u32(&bars->full[lane]), 1);
      mbar_init(smem_u32(&bars->empty[lane]), 2 * GROUPS);   // the two column blocks' warps of each group
    } else if (lane == S) {
      mbar_init(smem_u32(&bars->slab), 1);
      bars->abort = 0;
    }
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    for (int i = 0, t = tile, k = kk; i < first; ++i) {
      if (elect_one()) load_weights(i, t, k);
      __syncwarp();
      if (++k == p.k_iters) k = 0, ++t;
    }
    pdl_launch_dependents();
    if (cl > 1) {
      // rows r with r % cl == rank are finished here: their partial sums come from the cl - 1 other ranks
      const int rows = rank < p.m ? (p.m - rank + cl - 1) / cl : 0;
      if (rows && elect_one()) mbar_expect_tx(smem_u32(&bars->slab), (uint32_t)(rows * (cl - 1) * TILE_N * 4));
      __syncwarp();
    }
  }
  __syncthreads();
  if (cl > 1) cluster_arrive_relaxed();   // (the barriers' initialisation was released by fence.mbarrier_init)
  auto first_acts = [&]() {
    pdl_wait_prior_grid();
    for (int j = 0, ka = kk; j < first; ++j) {
      if (elect_one()) load_acts(j, ka);
      __syncwarp();
      if (++ka == p.k_iters) ka = 0;
    }
  };
  if (Cfg::PRODUCER && warp == NW) {
    // =========================================================== TMA producer
    first_acts();
    int i = first, t = (kk + first) / p.k_iters, k = kk + first - t * p.k_iters;
    t += tile;
    for (; i < total; ++i) {
      const int st = i % S;
      if (!warp_wait(smem_u32(&bars->empty[st]), ((i / S) & 1) ^ 1, abort, p.wait_ns)) { give_up(p, abort, 41); break; }
      if (elect_one()) {
        load_weights(st, t, k);
        load_acts(st, k);
      }
      __syncwarp();
      if (++k == p.k_iters) k = 0, ++t;
    }
    if (*abort) {   // unwinding: let the copies in flight land before the CTA may end
      volatile int never = 0;
      for (int j = max(0, i - S); j < i; ++j) mbar_wait(smem_u32(&bars->full[j % S]), (j / S) & 1, &never, 200000000ull);
    }
    if (cl > 1) cluster_wait();
    return;
  }
  if (!Cfg::PRODUCER) {
    if (warp == 0) first_acts();
    pdl_wait_prior_grid();                // (every requesting warp orders itself behind the previous kernel)
  }

  // =========================================================== consumers: warp = (64-column block b, k-lane lk); the lanes
  // take the CTA's 128-k groups in turn
  const int b = warp & 1, lk = warp >> 1;
  const uint32_t w_off = smem_u32(sW) + b * 512 + lane * 16;
  // ldmatrix row addresses.  MT = 1: matrices (k 0-7), (8-15), (16-23), (24-31) of two 16-k steps; MT = 2: (rows 0-7, k 0-7),
  // (0-7, 8-15), (8-15, 0-7), (8-15, 8-15) of one 16-k step
  const int ar = (lane & 7) + (MT > 1 ? (lane >> 4) * 8 : 0);
  const uint32_t ak = MT > 1 ? (lane >> 3) & 1 : lane >> 3;      // 16-byte column of the first step
  const uint32_t a_off = smem_u32(sA) + ar * 128;
  uint32_t a_col[MT > 1 ? 4 : 2];
#pragma unroll
  for (int q = 0; q < (MT > 1 ? 4 : 2); ++q) a_col[q] = (((MT > 1 ? 2 : 4) * q + ak) ^ (uint32_t)(ar & 7)) << 4;
  const uint32_t s_off = smem_u32(sS) + b * 128 + (lane >> 2) * 16;
  // its cells in the reduction buffer: rows 2 (lane % 4), + 1 (+ 8 t), columns 64 b + lane / 4 + 8 x
  const int red_off = (2 * (lane & 3)) * Cfg::RED_LD + b * 64 + (lane >> 2);

  bool first_segment = true;
  int g = lk;                                  // this warp's next 128-k group, counted over the CTA's stages
  // No producer warp (128-k stages only): the b = 0 warp of a k-lane requests, when it comes to group g, stage g - 4 + S into
  // the slot that both of the lane's warps have read in their previous turn.
  static_assert(S * GROUPS % LANES == 0, "a slot is always read by the same lane, which sees each phase of its barriers");
  static_assert(Cfg::PRODUCER || (GROUPS == 1 && S > LANES), "the slot of the previous turn");
  int rq_tile = 0, rq_kk = 0, rq_end = first;   // ...; one past the last stage that the lane may have in flight
  if (!Cfg::PRODUCER) {
    rq_tile = (kk + S + lk) / p.k_iters;
    rq_kk = kk + S + lk - rq_tile * p.k_iters;
    rq_tile += tile;
  }
  for (int done = 0; done < total; ++tile, kk = 0) {
    const int n0 = tile * TILE_N;
    const int kend = min(p.k_iters, kk + (total - done)), end = done + (kend - kk);
    float acc[4][MT][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][t][e] = 0.f;

    for (; g < end * GROUPS; g += LANES) {
      const int i = g / GROUPS, h = g % GROUPS, st = i % S;
      if (!Cfg::PRODUCER && b == 0 && g >= LANES && g - LANES + S < total) {
        const int j = g - LANES, slot = j % S;
        if (!warp_wait(smem_u32(&bars->empty[slot]), (j / S) & 1, abort, p.wait_ns)) { give_up(p, abort, 41); break; }
        if (elect_one()) {
          load_weights(slot, rq_tile, rq_kk);
          load_acts(slot, rq_kk);
        }
        __syncwarp();
        rq_end = j + S + 1;
        for (rq_kk += LANES; rq_kk >= p.k_iters; rq_kk -= p.k_iters) ++rq_tile;
      }
      if (!warp_wait(smem_u32(&bars->full[st]), (i / S) & 1, abort, p.wait_ns)) { give_up(p, abort, 42); break; }
      float tmp[4][MT][4];
      float(&d)[4][MT][4] = GROUPED ? tmp : acc;
      const uint32_t wb = w_off + st * Cfg::W_BYTES + h * 8192, ab = a_off + st * Cfg::A_BYTES + h * (2 * Cfg::ROWS * 128);
      uint32_t bf[4];
#pragma unroll
      for (int q = 0; q < 8; ++q) {   // 16-k steps
        uint32_t w[4];
        lds128(w, wb + q * 1024);
        if (MT > 1)
          ldmatrix_x4(bf, ab + (q >> 2) * (Cfg::ROWS * 128) + a_col[q & 3]);
        else if ((q & 1) == 0)
          ldmatrix_x4(bf, ab + (q >> 2) * (Cfg::ROWS * 128) + a_col[(q >> 1) & 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t a[4];
          dequant_word<false>(w[j], __half2(), a[0], a[2]);
          dequant_word<false>(w[j] >> 8, __half2(), a[1], a[3]);
#pragma unroll
          for (int t = 0; t < MT; ++t)
            mma_16816(d[j][t], a, bf[2 * (MT > 1 ? t : q & 1)], bf[2 * (MT > 1 ? t : q & 1) + 1], GROUPED && q == 0);
        }
      }
      uint32_t sv[4];
      if (GROUPED) lds128(sv, s_off + st * Cfg::S_BYTES + h * 256);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars->empty[st]));
      if (GROUPED) {
        // (q - 8) is exact in fp16: the MMAs sum exact integer-weight products per 128-k group, and the fp16 scale goes on
        // in fp32, as in the tcgen05 kernel for these batches
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // scales of columns 16 j + lane / 4, + 8
          const float2 s = __half22float2(*reinterpret_cast<const __half2 *>(&sv[j]));
#pragma unroll
          for (int t = 0; t < MT; ++t) {
            acc[j][t][0] = fmaf(s.x, tmp[j][t][0], acc[j][t][0]);
            acc[j][t][1] = fmaf(s.x, tmp[j][t][1], acc[j][t][1]);
            acc[j][t][2] = fmaf(s.y, tmp[j][t][2], acc[j][t][2]);
            acc[j][t][3] = fmaf(s.y, tmp[j][t][3], acc[j][t][3]);
          }
        }
      }
    }
    done = end;

    // ---- sum over the k-lanes of the CTA, through shared memory
    // (cluster form: every stage has been consumed, the ring is free; stream-K form: the previous tile's sums have been read)
    if (cl > 1 || !first_segment) bar_sync(1, NW * 32);
    first_segment = false;
    auto each = [&](float *dst, auto f) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) f(dst[red_off + (8 * t + (e & 1)) * Cfg::RED_LD + 16 * j + 8 * (e >> 1)], acc[j][t][e]);
    };
    if (cl > 1 || Cfg::SK_LANES == LANES) {
      each(red + lk * Cfg::RED_LANE, [](float &x, float v) { x = v; });
    } else {
      if (lk == 0) each(red, [](float &x, float v) { x = v; });
#pragma unroll 1
      for (int l = 1; l < LANES; ++l) {
        bar_sync(1, NW * 32);
        if (lk == l) each(red, [](float &x, float v) { x += v; });
      }
    }
    bar_sync(1, NW * 32);
    if (cl > 1) cluster_wait();           // every rank's barrier exists
    pdl_wait_prior_grid();                // C and the scratch may be in use by the previous kernel until here
    // warp w takes rows w, w + NW, ..., lane L columns 4 L .. 4 L + 3
    auto row_sum = [&](int row) {
      const float *src = red + row * Cfg::RED_LD + 4 * lane;
      float4 v = *reinterpret_cast<const float4 *>(src);
      const int lanes = cl > 1 ? LANES : Cfg::SK_LANES;
#pragma unroll
      for (int l = 1; l < LANES; ++l) {
        if (l >= lanes) break;
        const float4 x = *reinterpret_cast<const float4 *>(src + l * Cfg::RED_LANE);
        v.x += x.x, v.y += x.y, v.z += x.z, v.w += x.w;
      }
      return v;
    };
    if (cl > 1) {
      for (int row = warp; row < p.m; row += NW) {
        const int owner = row % cl;
        if (owner == rank) continue;
        // to the rank that finishes this row; slab: [row / cl][sender, without the owner][128]
        const int slot = (row / cl) * (cl - 1) + (rank < owner ? rank : rank - 1);
        st_async_f4(map_to_cta(smem_u32(slab + slot * TILE_N + 4 * lane), owner), row_sum(row), map_to_cta(smem_u32(&bars->slab), owner));
      }
      // A rank stays until its rows are complete: nothing may arrive in a CTA that has left.  (Hence a limit longer than any
      // other; a rank that gave up sends all the same.)
      if (rank < p.m && !warp_wait_cluster(smem_u32(&bars->slab), 0, 8 * p.wait_ns)) { give_up(p, abort, 43); break; }
    }
    // stream-K: CTAs cta + 1 .. cta + pieces hold the rest of a split tile
    const bool finisher = cl > 1 || kk == 0;
    const int pieces = cl == 1 && finisher && kend < p.k_iters ? ((tile + 1) * p.k_iters - 1) / p.iters_per_cta - cta : 0;
    for (int row = warp; row < p.m; row += NW) {
      if (cl > 1 && row % cl != rank) continue;
      float4 v = row_sum(row);
      if (!finisher) {
        st_slot4(p.partials + ((size_t)cta * Cfg::ROWS + row) * TILE_N + 4 * lane, v);
        continue;
      }
      for (int o = 0; o < cl - 1; ++o) {
        const float4 x = *reinterpret_cast<const float4 *>(slab + ((row / cl) * (cl - 1) + o) * TILE_N + 4 * lane);
        v.x += x.x, v.y += x.y, v.z += x.z, v.w += x.w;
      }
      if (pieces > 0 && !fold_slots4(v, p.partials + (((size_t)cta + 1) * Cfg::ROWS + row) * TILE_N + 4 * lane, Cfg::ROWS * TILE_N, pieces,
                                     abort, p.wait_ns)) {
        give_up(p, abort, 44);
        break;
      }
      __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
      if (!GROUPED) {   // per-channel scale after the fp16 convert (marlin_cute_trait.h:764-769)
        __half sc[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int col = n0 + 4 * lane + e, c32 = col & 31;
          sc[e] = p.s[col - c32 + 8 * ((c32 & 7) >> 1) + 2 * (c32 >> 3) + (c32 & 1)];
        }
        lo = __hmul2(lo, __halves2half2(sc[0], sc[1]));
        hi = __hmul2(hi, __halves2half2(sc[2], sc[3]));
      }
      const uint2 out = make_uint2(*reinterpret_cast<uint32_t *>(&lo), *reinterpret_cast<uint32_t *>(&hi));
      const size_t at = (size_t)row * p.c_ld + p.c_col0 + n0 + 4 * lane;
      *reinterpret_cast<uint2 *>(p.C + at) = out;
      if (p.C2) *reinterpret_cast<uint2 *>(p.C2 + at) = out;
      for (int x = 0; x < p.n_extra; ++x) *reinterpret_cast<uint2 *>(p.C_extra[x] + at) = out;   // the other ranks' buffers
    }
  }
  if (!Cfg::PRODUCER && b == 0 && *abort) {   // unwinding, as the producer does; a lane that ran to its end has nothing in flight
    volatile int never = 0;
    for (; g < rq_end; g += LANES) mbar_wait(smem_u32(&bars->full[g % S]), (g / S) & 1, &never, 200000000ull);
  }
}

}  // namespace w4a16
