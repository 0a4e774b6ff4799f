// Tensor-core products of float32-accurate operands, shared by the single track and by the
// general-shape triangle ops.
//
// An operand is a sum of bf16 pieces: one piece when the values are bf16 already, three when
// they are float32 (hi + mid + lo carry all 24 significand bits). The product is the sum of
// the piece products that matter - every pair down to 2^-16 of the leading one:
//   1 x 1: hi.hi        3 x 1: lo.hi, mid.hi, hi.hi       3 x 3: the six with i + j <= 2
//
// The tensor core truncates when it adds to its float32 accumulator, so every accumulation
// step costs a biased half ulp of the running sum (one accumulator for all terms of K = 384
// measured 3.2e-6 against float64, four times a float32 fma chain). The small terms therefore
// have an accumulator of their own, where that half ulp is 2^-8 smaller, and the leading term
// alternates between NMAIN accumulators; the epilogue adds them in float32.
//
// Single bf16 pieces have one accumulator for all of K. Against float64 without any rounding the
// triangle ops are as far off as with float32 fma chains on the CUDA cores: 7.46e-3 (multiplication)
// and 7.1e-3 (attention) of the result at 384 channels, equal to 3e-5 of that on average and to 2e-4
// in every case of 48 to 311 tokens; it is the bf16 roundings that count. Against the same bf16
// roundings with exact sums between them more results round the other way: of the 384-channel
// multiplication 7.9 % instead of 6.1, of the attention 6.0 instead of 4.4; at 64 channels 1.65
// instead of 1.6 and 0.69 instead of 0.63.
//
// piece_gemm_kernel: persistent, tiles of 128 x BN.
//   warp 0       TMA producer: per k step of 64 every piece of A [128][64] and of B [BN][64],
//                each K-major (activations) or MN-major (weights as stored, [in][out])
//   warp 1       MMA issuer
//   warps 4-     epilogue (policy code): EPI warps, EPI / 4 per TMEM lane quarter, each with its
//                share of the columns, 16 at a time
// The epilogues (conversions, gates, scattered stores) are latency-bound: a policy asks for two
// CTAs per SM where its tile fits twice, or for more epilogue warps where it does not.
// A tile has one or two segments (two products with operands of their own, in neighbouring
// TMEM columns), and its accumulators are double-buffered where they fit, so that the epilogue
// of one tile overlaps the products of the next. With few tiles K is split: each split writes its own partial.
// The device status word is asked for beside a CTA's last epilogue alone: by every epilogue warp at every tile it was one
// word that all SMs loaded two times a nanosecond (four updates of four 200-token templates 586 -> 573 us).
#pragma once
#include "host.cuh"
#include "tc.cuh"

namespace b200 {

constexpr int GEMM_BM = 128, GEMM_BK = 64;
constexpr int GEMM_A_BYTES = GEMM_BM * GEMM_BK * 2;  // one piece of one k step

// v = hi + mid + lo
__device__ __forceinline__ void split3(float v, __nv_bfloat16& hi, __nv_bfloat16& mid, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(v);
  const float r = v - __bfloat162float(hi);
  mid = __float2bfloat16_rn(r);
  lo = __float2bfloat16_rn(r - __bfloat162float(mid));
}
// v - (the pair's two values), one instruction each (8 % of
// the bf16 attention core, against two to unpack and half a packed one).
__device__ __forceinline__ float2 less_bf16x2(float2 v, uint32_t w) {
  float2 r;
  asm("{\n"
      " .reg .b16 lo, hi, m;\n"
      " mov.b32 {lo, hi}, %2;\n"
      " mov.b16 m, 0xBF80;\n"
      " fma.rn.f32.bf16 %0, lo, m, %3;\n"
      " fma.rn.f32.bf16 %1, hi, m, %4;\n"
      "}\n"
      : "=f"(r.x), "=f"(r.y)
      : "r"(w), "f"(v.x), "f"(v.y));
  return r;
}
// split3 for two neighbouring values, packed (256-token float32 stack 909 -> 904 us against unpacked pieces, the same bits).
__device__ __forceinline__ void split3x2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(a, b);
  const float2 r = less_bf16x2(make_float2(a, b), hi);
  mid = pack_bf16x2(r.x, r.y);
  const float2 q = less_bf16x2(r, mid);
  lo = pack_bf16x2(q.x, q.y);
}

template <int PA, int PB>
struct Terms;
template <>
struct Terms<1, 1> {
  static constexpr int N = 1;
  static __device__ constexpr int a(int) { return 0; }
  static __device__ constexpr int b(int) { return 0; }
};
template <>
struct Terms<3, 1> {
  static constexpr int N = 3;
  static __device__ constexpr int a(int t) { return 2 - t; }
  static __device__ constexpr int b(int) { return 0; }
};
template <>
struct Terms<3, 3> {
  static constexpr int N = 6;
  static __device__ constexpr int a(int t) { return t == 0 ? 2 : t == 1 ? 0 : t == 2 ? 1 : t == 3 ? 1 : 0; }
  static __device__ constexpr int b(int t) { return t == 0 ? 0 : t == 1 ? 2 : t == 2 ? 1 : t == 3 ? 0 : t == 4 ? 1 : 0; }
};

struct GemmMaps {
  CUtensorMap a[2], b[4];
};
struct GemmShape {
  int m_tiles, n_tiles, splits;
  int kb[2];  // k steps of 64 per segment
  int* status;
  // set by the launch: k steps of a split, and what tile numbers are divided by
  int per[2];
  Divisor by_splits, fast;  // (fast: tiles of the direction that successive tiles walk)
};

// What a policy P provides:
//   BN, PA, PB, NSEG, NMAIN, A_MN, B_MN, M_FAST   shape constants (M_FAST: successive tiles walk m)
//   EPI, CTAS                                     epilogue warps, CTAs per SM
//   TURNS (with an operand resident)              whether the epilogue warps take a tile's columns in turn
//   struct Params                                 arguments
//   load_a / load_b(maps, params, seg, k, tile, piece, dst, bar)  one piece of one k step
//   Pre, prefetch(params, m_tile, n_tile, quarter, col0, col1, lane, pre)   what the epilogue reads from
//                     global memory, requested before the accumulators are waited for (or NoPrefetch)
//   epilogue(params, m_tile, n_tile, split, accumulators, quarter, col0, col1, lane, pre)   columns [col0, col1)
struct NoPrefetch {
  struct Pre {};
  template <class... A>
  static __device__ __forceinline__ void prefetch(const A&...) {}
};
template <class P>
constexpr int gemm_acc_count() {  // accumulators of one segment
  return P::NMAIN + (P::PA * P::PB > 1 ? 1 : 0);
}

// The accumulators of a finished tile, as the epilogue reads them.
template <class P>
struct Accum {
  uint32_t base;  // TMEM address of the warp's lanes, first column of the tile
  int used[P::NSEG];  // k steps of each segment: only so many leading-term accumulators were written
  // 16 columns starting at `col` of segment `seg`, one TMEM lane per thread
  __device__ __forceinline__ void load(int seg, int col, float (&v)[16]) const {
    constexpr int NACC = gemm_acc_count<P>();
    __syncwarp();  // (the callers' guards may have split the warp; TMEM loads are warp-wide)
    uint32_t r[NACC][16];
    const uint32_t t = base + seg * (NACC * P::BN) + col;
#pragma unroll
    for (int m = 0; m < NACC; ++m) tmem_ld16(t + m * P::BN, r[m]);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[0][e]);
#pragma unroll
    for (int m = 1; m < NACC; ++m) {
      if (m < P::NMAIN && m >= used[seg]) continue;
#pragma unroll
      for (int e = 0; e < 16; ++e) v[e] += __uint_as_float(r[m][e]);
    }
  }
};

// MN-major operand piece: `groups` boxes of 64 columns from `col` on, 64 rows of k.
__device__ __forceinline__ void gemm_load_mn(const CUtensorMap* m, uint8_t* dst, uint64_t* bar, int groups, int col, int k,
                                             int piece) {
  for (int g = 0; g < groups; ++g) tma_load_3d(dst + g * 8192, m, bar, col + g * 64, k, piece);
}

template <class P>
constexpr int gemm_stage_bytes() {
  return P::PA * GEMM_A_BYTES + P::PB * P::BN * 128;
}
template <class P>
constexpr int gemm_stages() {
  constexpr int fit = (P::CTAS == 1 ? 220 : 110) * 1024 / gemm_stage_bytes<P>();
  return fit > 6 ? 6 : fit;
}
template <class P>
constexpr int gemm_threads() {
  return 128 + P::EPI * 32;
}
template <class P>
constexpr int gemm_smem_bytes() {
  return gemm_stages<P>() * gemm_stage_bytes<P>() + 1024;
}

template <class P>
__global__ void __launch_bounds__(gemm_threads<P>(), P::CTAS)
piece_gemm_kernel(const __grid_constant__ GemmMaps maps, const GemmShape g, const typename P::Params ep) {
  constexpr int STAGES = gemm_stages<P>(), STAGE_BYTES = gemm_stage_bytes<P>();
  constexpr int SEG = gemm_acc_count<P>() * P::BN;  // accumulator columns of one segment
  constexpr int ACC = P::NSEG * SEG;                // and of one tile
  constexpr uint32_t NBUF = 2 * ACC <= 512 / P::CTAS ? 2 : 1;
  constexpr int USED = NBUF * ACC, TMEM_COLS = USED <= 64 ? 64 : USED <= 128 ? 128 : USED <= 256 ? 256 : 512;
  static_assert(NBUF * ACC <= 512 / P::CTAS && STAGES >= 2, "tile does not fit");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (warp == 0 && lane == 0) {
    for (int s = 0; s < P::NSEG; ++s) tma_prefetch_desc(&maps.a[s]);
    tma_prefetch_desc(&maps.b[0]);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {  // (one is spare without double buffering)
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], P::EPI);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  int status = -1;
  const uint32_t tmem_base = tmem_base_s;
  // (32-bit tile arithmetic: a 64-bit division costs a role several hundred cycles per tile)
  const uint32_t total = static_cast<uint32_t>(g.m_tiles) * g.n_tiles * g.splits;
  auto locate = [&](uint32_t tile, int& split, int& m_tile, int& n_tile) {
    const uint32_t whole = g.by_splits.quotient(tile);
    split = static_cast<int>(tile - whole * g.by_splits.d);
    tile = whole;
    const int hi = static_cast<int>(g.fast.quotient(tile)), lo = static_cast<int>(tile - hi * g.fast.d);
    m_tile = P::M_FAST ? lo : hi;
    n_tile = P::M_FAST ? hi : lo;
  };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      for (uint32_t tile = blockIdx.x; tile < total && alive; tile += gridDim.x) {
        int split, m_tile, n_tile;
        locate(tile, split, m_tile, n_tile);
        for (int seg = 0; seg < P::NSEG && alive; ++seg) {
          const int per = g.per[seg];
          const int k1 = min(g.kb[seg], (split + 1) * per);
          for (int kb = split * per; kb < k1; ++kb) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, g.status, ST_TIMEOUT_PRODUCER)) {
              alive = false;
              break;
            }
            uint8_t* sa = smem + stage * STAGE_BYTES;
            uint8_t* sb = sa + P::PA * GEMM_A_BYTES;
            mbar_expect_tx(&full_bar[stage], STAGE_BYTES);
            for (int pc = 0; pc < P::PA; ++pc)
              P::load_a(maps, ep, seg, kb * GEMM_BK, m_tile, pc, sa + pc * GEMM_A_BYTES, &full_bar[stage]);
            for (int pc = 0; pc < P::PB; ++pc)
              P::load_b(maps, ep, seg, kb * GEMM_BK, n_tile, pc, sb + pc * P::BN * 128, &full_bar[stage]);
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(GEMM_BM, P::BN) | (P::A_MN ? UMMA_A_MN : 0u) | (P::B_MN ? UMMA_B_MN : 0u);
      using T = Terms<P::PA, P::PB>;
      int stage = 0;
      uint32_t phase = 0, it = 0;
      bool alive = true;
      for (uint32_t tile = blockIdx.x; tile < total && alive; tile += gridDim.x, ++it) {
        const int split = static_cast<int>(tile - g.by_splits.quotient(tile) * g.by_splits.d);
        const uint32_t buf = it % NBUF, buf_phase = (it / NBUF) & 1;
        if (!mbar_wait(&acc_empty[buf], buf_phase ^ 1, g.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        for (int seg = 0; seg < P::NSEG && alive; ++seg) {
          const uint32_t d_seg = tmem_base + buf * ACC + seg * SEG;
          const int per = g.per[seg];
          const int k0 = split * per, k1 = min(g.kb[seg], (split + 1) * per);
          for (int kb = k0; kb < k1; ++kb) {
            if (!mbar_wait(&full_bar[stage], phase, g.status, ST_TIMEOUT_MMA)) {
              alive = false;
              break;
            }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
            const uint32_t sb = sa + P::PA * GEMM_A_BYTES;
#pragma unroll
            for (int t = 0; t < T::N; ++t) {
              const uint64_t adesc = P::A_MN ? umma_desc_mnmajor(sa + T::a(t) * GEMM_A_BYTES, 8192)
                                             : umma_desc_kmajor(sa + T::a(t) * GEMM_A_BYTES, 128);
              const uint64_t bdesc = P::B_MN ? umma_desc_mnmajor(sb + T::b(t) * P::BN * 128, 8192)
                                             : umma_desc_kmajor(sb + T::b(t) * P::BN * 128, 128);
              const bool lead = t == T::N - 1;
              const uint32_t d_tmem = d_seg + (lead ? (kb - k0) % P::NMAIN : P::NMAIN) * P::BN;
              const int fresh = lead ? kb - k0 < P::NMAIN : (kb == k0 && t == 0);  // first product into it
#pragma unroll
              for (int k = 0; k < GEMM_BK / 16; ++k)
                umma_bf16_ss(d_tmem, umma_desc_advance(adesc, P::A_MN ? k * 2048 : k * 32),
                             umma_desc_advance(bdesc, P::B_MN ? k * 2048 : k * 32), idesc, !(fresh && k == 0));
            }
            umma_commit(&empty_bar[stage]);
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
        if (alive) umma_commit(&acc_full[buf]);
      }
    }
  } else if (warp >= 4) {
    const int quarter = warp & 3, part = (warp - 4) >> 2;
    constexpr int SHARE = P::BN / (P::EPI / 4);
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < total; tile += gridDim.x, ++it) {
      int split, m_tile, n_tile;
      locate(tile, split, m_tile, n_tile);
      const uint32_t buf = it % NBUF, buf_phase = (it / NBUF) & 1;
      typename P::Pre pre;
      P::prefetch(ep, m_tile, n_tile, quarter, part * SHARE, (part + 1) * SHARE, lane, pre);
      if (!mbar_wait(&acc_full[buf], buf_phase, g.status, ST_TIMEOUT_EPILOGUE)) {
        status = -1;
        break;
      }
      tc_fence_after();
      Accum<P> acc;
      acc.base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * ACC;
#pragma unroll
      for (int seg = 0; seg < P::NSEG; ++seg) {
        const int per = g.per[seg];
        acc.used[seg] = min(g.kb[seg], (split + 1) * per) - split * per;
      }
      if (tile + gridDim.x >= total) status = ask_status(g.status);  // (arrives during the last epilogue)
      P::epilogue(ep, m_tile, n_tile, split, acc, quarter, part * SHARE, (part + 1) * SHARE, lane, pre);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }

  settle(status, g.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

template <class P>
int launch_piece_gemm(const GemmMaps& maps, GemmShape g, const typename P::Params& ep, cudaStream_t stream, bool pdl) {
  g.status = device_status_word();
  B200_REQUIRE(g.status != nullptr, B200TRI_ERR_CUDA, "gemm: no current CUDA device");
  int rc = ensure_smem_limit(reinterpret_cast<const void*>(piece_gemm_kernel<P>), gemm_smem_bytes<P>());
  if (rc) return rc;
  const long long total = static_cast<long long>(g.m_tiles) * g.n_tiles * g.splits;
  B200_REQUIRE(total < (1ll << 32) - 1024, B200TRI_ERR_UNSUPPORTED, "gemm: too many tiles (%lld)", total);
  for (int seg = 0; seg < 2; ++seg) g.per[seg] = (g.kb[seg] + g.splits - 1) / g.splits;
  g.by_splits = Divisor(g.splits);
  g.fast = Divisor(P::M_FAST ? g.m_tiles : g.n_tiles);
  const long long slots = static_cast<long long>(P::CTAS) * sm_count();
  const unsigned grid = static_cast<unsigned>(total < slots ? total : slots);
  return launch(piece_gemm_kernel<P>, dim3(grid), dim3(gemm_threads<P>()), gemm_smem_bytes<P>(), stream, pdl, maps, g, ep);
}

// The same product with one operand resident: a CTA keeps the rows of a slow-direction tile (A, or
// with M_FAST the B tile that both segments share) for all its k steps and streams the other
// operand for a run of fast-direction tiles. A 128 x 128 tile reads 32 KiB per k step into the SM
// otherwise, 512 clocks for 256 of products; so it reads half. The resident k steps have barriers
// of their own and are refilled one by one behind the last tile's products.
// Gated projection, 65 536 pairs x 384 -> 768 channels: 104 -> 94 us; 160 000 x 64 -> 256: 72 -> 67;
// q, k, v and bias, 160 000 x 64: 56 -> 45 (wider ones where there are tiles enough: the rule is in generic.cu).
constexpr int RES_KB = 8, RES_STAGES = 8, RES_SLOTS = 16;  // most k steps kept, streamed stages, places of either
template <class P>
constexpr int gemm_res_bytes() {
  return P::M_FAST ? P::PB * P::BN * 128 : P::PA * GEMM_A_BYTES;
}
template <class P>
constexpr int gemm_stream_bytes() {
  return gemm_stage_bytes<P>() - gemm_res_bytes<P>();
}
template <class P>
int gemm_res_stages(int kb) {  // 0: does not fit
  const int left = 222 * 1024 - kb * gemm_res_bytes<P>();
  const int stages = kb > RES_KB || left < 0 ? 0 : left / gemm_stream_bytes<P>();
  return stages < 3 ? 0 : stages > RES_STAGES ? RES_STAGES : stages;
}
struct GemmRuns {
  int fast, log_parts, slots, stages;  // fast-direction tiles, runs they are cut into (log2), kept places, streamed stages
  uint32_t units;           // slow-direction tiles x parts
};

// KEPT_KB > 0: the stages hold the whole streamed operand (the weights) of so many k steps, which is loaded for a CTA's first
// unit and stays, and there are places for several units' k steps.
template <class P, int KEPT_KB>
__global__ void __launch_bounds__(gemm_threads<P>(), 1)
piece_gemm_resident_kernel(const __grid_constant__ GemmMaps maps, const GemmShape g, const GemmRuns runs,
                           const typename P::Params ep) {
  static_assert(P::CTAS == 1 && (P::M_FAST || P::NSEG == 1), "one operand for all segments");
  constexpr bool ONCE = KEPT_KB > 0;
  constexpr int RES = gemm_res_bytes<P>(), STREAM = gemm_stream_bytes<P>();
  constexpr int SEG = gemm_acc_count<P>() * P::BN, ACC = P::NSEG * SEG;
  constexpr uint32_t NBUF = 2 * ACC <= 512 ? 2 : 1;
  constexpr int USED = NBUF * ACC, TMEM_COLS = USED <= 64 ? 64 : USED <= 128 ? 128 : USED <= 256 ? 256 : 512;
  static_assert(NBUF * ACC <= 512, "tile does not fit");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int kbs = ONCE ? KEPT_KB : g.kb[0], slots = ONCE ? runs.slots : kbs, stages = runs.stages;
  uint8_t* ring = smem + slots * RES;
  __shared__ uint64_t res_full[RES_SLOTS], res_empty[RES_SLOTS], full_bar[RES_SLOTS], empty_bar[RES_SLOTS], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    for (int s = 0; s < P::NSEG; ++s) tma_prefetch_desc(&maps.a[s]);
    tma_prefetch_desc(&maps.b[0]);
    for (int s = 0; s < RES_SLOTS; ++s) {
      mbar_init(&res_full[s], 1);
      mbar_init(&res_empty[s], 1);
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], P::EPI);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  int status = -1;
  const uint32_t tmem_base = tmem_base_s;
  // the place of a unit's k step, counted from that of its first one, and the first place of the next unit
  auto place = [&](int kept, int kb) { return !ONCE ? kb : kept + kb < slots ? kept + kb : kept + kb - slots; };
  auto next_kept = [&](int& kept, uint32_t& round) {
    if (!ONCE) {
      round ^= 1;
      return;
    }
    kept += kbs;
    if (kept >= slots) {
      kept -= slots;
      round ^= 1;
    }
  };
  auto locate = [&](uint32_t unit, int& slow, int& f0, int& f1) {
    const uint32_t s = unit >> runs.log_parts, part = unit - (s << runs.log_parts);
    slow = s;
    f0 = part * runs.fast >> runs.log_parts;
    f1 = (part + 1) * runs.fast >> runs.log_parts;
  };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0, kept = 0;  // kept: slot of the unit's first k step
      uint32_t phase = 0, round = 0;
      bool alive = true;
      for (uint32_t unit = blockIdx.x; unit < runs.units && alive; unit += gridDim.x, next_kept(kept, round)) {
        int slow, f0, f1;
        locate(unit, slow, f0, f1);
        for (int f = f0; f < f1 && alive; ++f) {
          const int m_tile = P::M_FAST ? f : slow, n_tile = P::M_FAST ? slow : f;
          for (int seg = 0; seg < P::NSEG && alive; ++seg)
            for (int kb = 0; kb < kbs; ++kb) {
              if (f == f0 && seg == 0) {
                const int slot = place(kept, kb);
                if (!mbar_wait(&res_empty[slot], round ^ (slot >= kept), g.status, ST_TIMEOUT_PRODUCER)) {
                  alive = false;
                  break;
                }
                mbar_expect_tx(&res_full[slot], RES);
                for (int pc = 0; pc < (P::M_FAST ? P::PB : P::PA); ++pc) {
                  if (P::M_FAST)
                    P::load_b(maps, ep, 0, kb * GEMM_BK, n_tile, pc, smem + slot * RES + pc * P::BN * 128, &res_full[slot]);
                  else
                    P::load_a(maps, ep, 0, kb * GEMM_BK, m_tile, pc, smem + slot * RES + pc * GEMM_A_BYTES, &res_full[slot]);
                }
              }
              if (ONCE && unit != blockIdx.x) continue;
              if (!mbar_wait(&empty_bar[stage], phase ^ 1, g.status, ST_TIMEOUT_PRODUCER)) {
                alive = false;
                break;
              }
              mbar_expect_tx(&full_bar[stage], STREAM);
              for (int pc = 0; pc < (P::M_FAST ? P::PA : P::PB); ++pc) {
                if (P::M_FAST)
                  P::load_a(maps, ep, seg, kb * GEMM_BK, m_tile, pc, ring + stage * STREAM + pc * GEMM_A_BYTES, &full_bar[stage]);
                else
                  P::load_b(maps, ep, seg, kb * GEMM_BK, n_tile, pc, ring + stage * STREAM + pc * P::BN * 128, &full_bar[stage]);
              }
              if (++stage == stages) {
                stage = 0;
                phase ^= 1;
              }
            }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(GEMM_BM, P::BN) | (P::A_MN ? UMMA_A_MN : 0u) | (P::B_MN ? UMMA_B_MN : 0u);
      using T = Terms<P::PA, P::PB>;
      int stage = 0, kept = 0;
      uint32_t phase = 0, it = 0, round = 0;
      bool alive = true;
      for (uint32_t unit = blockIdx.x; unit < runs.units && alive; unit += gridDim.x, next_kept(kept, round)) {
        int slow, f0, f1;
        locate(unit, slow, f0, f1);
        for (int f = f0; f < f1 && alive; ++f, ++it) {
          const uint32_t buf = it % NBUF, buf_phase = (it / NBUF) & 1;
          if (!mbar_wait(&acc_empty[buf], buf_phase ^ 1, g.status, ST_TIMEOUT_MMA)) {
            alive = false;
            break;
          }
          tc_fence_after();
#pragma unroll
          for (int seg = 0; seg < P::NSEG && alive; ++seg)
#pragma unroll
            for (int kb = 0; kb < kbs; ++kb) {
              const int slot = place(kept, kb);
              if ((f == f0 && seg == 0 && !mbar_wait(&res_full[slot], round ^ (slot < kept), g.status, ST_TIMEOUT_MMA)) ||
                  ((!ONCE || unit == blockIdx.x) && !mbar_wait(&full_bar[stage], phase, g.status, ST_TIMEOUT_MMA))) {
                alive = false;
                break;
              }
              tc_fence_after();
              const uint32_t resident = smem_u32(smem + slot * RES), streamed = smem_u32(ring + stage * STREAM);
              const uint32_t sa = P::M_FAST ? streamed : resident, sb = P::M_FAST ? resident : streamed;
#pragma unroll
              for (int t = 0; t < T::N; ++t) {
                const uint64_t adesc = P::A_MN ? umma_desc_mnmajor(sa + T::a(t) * GEMM_A_BYTES, 8192)
                                               : umma_desc_kmajor(sa + T::a(t) * GEMM_A_BYTES, 128);
                const uint64_t bdesc = P::B_MN ? umma_desc_mnmajor(sb + T::b(t) * P::BN * 128, 8192)
                                               : umma_desc_kmajor(sb + T::b(t) * P::BN * 128, 128);
                const bool lead = t == T::N - 1;
                const uint32_t d_tmem = tmem_base + buf * ACC + seg * SEG + (lead ? kb % P::NMAIN : P::NMAIN) * P::BN;
                const int fresh = lead ? kb < P::NMAIN : (kb == 0 && t == 0);  // first product into it
#pragma unroll
                for (int k = 0; k < GEMM_BK / 16; ++k)
                  umma_bf16_ss(d_tmem, umma_desc_advance(adesc, P::A_MN ? k * 2048 : k * 32),
                               umma_desc_advance(bdesc, P::B_MN ? k * 2048 : k * 32), idesc, !(fresh && k == 0));
              }
              if (!ONCE) umma_commit(&empty_bar[stage]);
              if (f == f1 - 1 && seg == P::NSEG - 1) umma_commit(&res_empty[slot]);
              if (++stage == stages) {
                stage = 0;
                phase ^= 1;
              }
            }
          if (alive) umma_commit(&acc_full[buf]);
        }
      }
    }
  } else if (warp >= 4) {
    const int quarter = warp & 3;
    constexpr int PARTS = P::EPI / 4, SHARE = P::BN / PARTS;
    uint32_t it = 0;
    bool alive = true;
    for (uint32_t unit = blockIdx.x; unit < runs.units && alive; unit += gridDim.x) {
      int slow, f0, f1;
      locate(unit, slow, f0, f1);
      for (int f = f0; f < f1; ++f, ++it) {
        const int m_tile = P::M_FAST ? f : slow, n_tile = P::M_FAST ? slow : f;
        const uint32_t buf = it % NBUF, buf_phase = (it / NBUF) & 1;
        const int part = static_cast<int>((warp - 4) / 4 + (P::TURNS ? it + it / PARTS : 0)) % PARTS;
        typename P::Pre pre;
        P::prefetch(ep, m_tile, n_tile, quarter, part * SHARE, (part + 1) * SHARE, lane, pre);
        if (!mbar_wait(&acc_full[buf], buf_phase, g.status, ST_TIMEOUT_EPILOGUE)) {
          alive = false;
          status = -1;
          break;
        }
        tc_fence_after();
        Accum<P> acc;
        acc.base = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * ACC;
#pragma unroll
        for (int seg = 0; seg < P::NSEG; ++seg) acc.used[seg] = kbs;
        if (f == f1 - 1 && unit + gridDim.x >= runs.units) status = ask_status(g.status);  // (arrives during the epilogue)
        P::epilogue(ep, m_tile, n_tile, 0, acc, quarter, part * SHARE, (part + 1) * SHARE, lane, pre);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
    }
  }

  settle(status, g.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// The caller has checked gemm_res_stages<P>(kb) and that all segments have g.kb[0] k steps.
template <class P>
int launch_piece_gemm_resident(const GemmMaps& maps, GemmShape g, const typename P::Params& ep, cudaStream_t stream, bool pdl) {
  g.status = device_status_word();
  B200_REQUIRE(g.status != nullptr, B200TRI_ERR_CUDA, "gemm: no current CUDA device");
  const int slow = P::M_FAST ? g.n_tiles : g.m_tiles;
  GemmRuns r = {P::M_FAST ? g.m_tiles : g.n_tiles, 0, g.kb[0], gemm_res_stages<P>(g.kb[0]), 0};
  // enough runs that the last wave matters little, of at least two tiles, or of one where they all run at once
  // (64 tokens: template 81.0 -> 77.3 us, float32 stack 153.5 -> 142.1)
  auto runs_of = [&](int log) { return static_cast<long long>(slow) << log; };
  while ((runs_of(r.log_parts) < 6ll * sm_count() && r.fast >> r.log_parts >= 4) ||
         (runs_of(r.log_parts + 1) <= sm_count() && r.fast >> r.log_parts >= 2))
    ++r.log_parts;
  const long long units = runs_of(r.log_parts);
  B200_REQUIRE(units < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "gemm: too many tiles (%lld)", units);
  r.units = static_cast<uint32_t>(units);
  const unsigned grid = static_cast<unsigned>(units < sm_count() ? units : sm_count());
  auto go = [&](auto kernel) {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), 223 * 1024);
    if (rc) return rc;
    const size_t smem = static_cast<size_t>(r.slots) * gemm_res_bytes<P>() + r.stages * gemm_stream_bytes<P>() + 1024;
    return launch(kernel, dim3(grid), dim3(gemm_threads<P>()), smem, stream, pdl, maps, g, r, ep);
  };
  // Weights of up to 16 k steps stay where two units' rows fit beside them. Streamed, all SMs fetched the same few lines
  // from L2 at a time (64 rows of 16 bytes for a bias of 4 heads), and loads and products alone took 28 of the 41 us of the
  // projection of four 200-token templates; now it takes 29 (four updates 568 -> 551 us, 320 tokens 407 -> 392).
  if constexpr (P::PA * P::PB == 1) {
    const int all = r.fast * P::NSEG * g.kb[0];
    const int left = (222 * 1024 - all * gemm_stream_bytes<P>()) / gemm_res_bytes<P>();
    if (g.kb[0] <= 2 && r.log_parts == 0 && all <= RES_SLOTS && left >= 2 * g.kb[0]) {
      const int most = 4 * g.kb[0] < RES_SLOTS ? 4 * g.kb[0] : RES_SLOTS;
      r.slots = left < most ? left : most;
      r.stages = all;
      if (g.kb[0] == 1) return go(piece_gemm_resident_kernel<P, 1>);
      return go(piece_gemm_resident_kernel<P, 2>);
    }
  }
  return go(piece_gemm_resident_kernel<P, 0>);
}

// Activations: bf16 pieces [pieces][rows][k], row pitch `pitch` elements (a multiple of 8);
// `box_rows` rows per load.
inline int gemm_map_kmajor(CUtensorMap* out, const void* base, int pieces, long long rows, int k, long long pitch,
                           int box_rows) {
  const uint64_t dims[3] = {static_cast<uint64_t>(k), static_cast<uint64_t>(rows), static_cast<uint64_t>(pieces)};
  const uint64_t str[2] = {static_cast<uint64_t>(pitch) * 2, static_cast<uint64_t>(pitch) * rows * 2};
  const uint32_t box[3] = {GEMM_BK, static_cast<uint32_t>(box_rows), 1};
  return make_tmap(out, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
}
// Weights as stored, [pieces][k][n] with row pitch `pitch` (a multiple of 8), read as MN-major tiles.
inline int gemm_map_mnmajor(CUtensorMap* out, const void* base, int k, int n, long long pitch, int pieces = 1) {
  const uint64_t dims[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k), static_cast<uint64_t>(pieces)};
  const uint64_t str[2] = {static_cast<uint64_t>(pitch) * 2, static_cast<uint64_t>(pitch) * k * 2};
  const uint32_t box[3] = {64, GEMM_BK, 1};
  return make_tmap(out, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
}

}  // namespace b200
