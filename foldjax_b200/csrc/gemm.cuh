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
// piece_gemm_kernel: persistent, one CTA per SM, tiles of 128 x BN.
//   warp 0       TMA producer: per k step of 64 every piece of A [128][64] (K-major) and of B,
//                either K-major [BN][64] or MN-major [64][BN] (weights as stored, [in][out])
//   warp 1       MMA issuer
//   warps 4-11   epilogue (policy code), two warps per TMEM lane quarter
// A tile has one or two segments (two products with operands of their own, in neighbouring
// TMEM columns), and its accumulators are double-buffered where they fit, so that the epilogue
// of one tile overlaps the products of the next. With few tiles K is split: each split writes its own partial.
#pragma once
#include "host.cuh"
#include "tc.cuh"

namespace b200 {

constexpr int GEMM_BM = 128, GEMM_BK = 64;
constexpr int GEMM_A_BYTES = GEMM_BM * GEMM_BK * 2;  // one piece of one k step
constexpr int GEMM_EPI_WARPS = 8;
constexpr int GEMM_THREADS = 128 + GEMM_EPI_WARPS * 32;

// v = hi + mid + lo
__device__ __forceinline__ void split3(float v, __nv_bfloat16& hi, __nv_bfloat16& mid, __nv_bfloat16& lo) {
  hi = __float2bfloat16_rn(v);
  const float r = v - __bfloat162float(hi);
  mid = __float2bfloat16_rn(r);
  lo = __float2bfloat16_rn(r - __bfloat162float(mid));
}
// The same for two neighbouring values, packed.
__device__ __forceinline__ void split3x2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(a, b);
  const float ra = a - bf16_lo(hi), rb = b - bf16_hi(hi);
  mid = pack_bf16x2(ra, rb);
  lo = pack_bf16x2(ra - bf16_lo(mid), rb - bf16_hi(mid));
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
};

// What a policy P provides:
//   BN, PA, PB, NSEG, NMAIN, B_MN              shape constants
//   struct Params                              epilogue arguments
//   b_map(seg, n_tile, g, params), b_col(...)  which B map and column group g (64 wide, MN-major)
//                                              or row block (K-major, g = 0) of a tile reads
//   epilogue(params, m_tile, n_tile, split, accumulators, quarter, half, lane)
template <class P>
constexpr int gemm_acc_count() {  // accumulators of one segment
  return P::NMAIN + (P::PA * P::PB > 1 ? 1 : 0);
}

// The accumulators of a finished tile, as the epilogue reads them.
template <class P>
struct Accum {
  uint32_t base;  // TMEM address of the warp's lanes, first column of the tile
  int used;       // leading-term accumulators that were written
  // 32 columns starting at `col` of segment `seg`, one TMEM lane per thread
  __device__ __forceinline__ void load(int seg, int col, float (&v)[32]) const {
    constexpr int NACC = gemm_acc_count<P>();
    uint32_t r[32];
    const uint32_t t = base + seg * (NACC * P::BN) + col;
    tmem_ld32(t, r);
    tmem_ld_wait();
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = __uint_as_float(r[e]);
#pragma unroll
    for (int m = 1; m < NACC; ++m) {
      if (m < P::NMAIN && m >= used) continue;
      tmem_ld32(t + m * P::BN, r);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 32; ++e) v[e] += __uint_as_float(r[e]);
    }
  }
};

template <class P>
constexpr int gemm_stage_bytes() {
  return P::PA * GEMM_A_BYTES + P::PB * P::BN * 128;
}
template <class P>
constexpr int gemm_stages() {
  return (220 * 1024) / gemm_stage_bytes<P>() > 6 ? 6 : (220 * 1024) / gemm_stage_bytes<P>();
}
template <class P>
constexpr int gemm_smem_bytes() {
  return gemm_stages<P>() * gemm_stage_bytes<P>() + 1024;
}

template <class P>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
piece_gemm_kernel(const __grid_constant__ GemmMaps maps, const GemmShape g, const typename P::Params ep) {
  constexpr int STAGES = gemm_stages<P>(), STAGE_BYTES = gemm_stage_bytes<P>();
  constexpr int SEG = gemm_acc_count<P>() * P::BN;  // accumulator columns of one segment
  constexpr int ACC = P::NSEG * SEG;                // and of one tile
  constexpr uint32_t NBUF = 2 * ACC <= 512 ? 2 : 1;
  constexpr int USED = NBUF * ACC, TMEM_COLS = USED <= 64 ? 64 : USED <= 128 ? 128 : USED <= 256 ? 256 : 512;
  static_assert(ACC <= 512 && STAGES >= 2, "tile does not fit");
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
      mbar_init(&acc_empty[b], GEMM_EPI_WARPS);
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
  const uint32_t tmem_base = tmem_base_s;
  const long long total = static_cast<long long>(g.m_tiles) * g.n_tiles * g.splits;

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      for (long long tile = blockIdx.x; tile < total && alive; tile += gridDim.x) {
        const int split = static_cast<int>(tile % g.splits);
        const int n_tile = static_cast<int>((tile / g.splits) % g.n_tiles);
        const int m_tile = static_cast<int>(tile / g.splits / g.n_tiles);
        for (int seg = 0; seg < P::NSEG && alive; ++seg) {
          const int per = (g.kb[seg] + g.splits - 1) / g.splits;
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
              tma_load_3d(sa + pc * GEMM_A_BYTES, &maps.a[seg], &full_bar[stage], kb * GEMM_BK, m_tile * GEMM_BM, pc);
            for (int pc = 0; pc < P::PB; ++pc) {
              if (P::B_MN) {
                for (int grp = 0; grp < P::BN / 64; ++grp)
                  tma_load_3d(sb + pc * P::BN * 128 + grp * 8192, &maps.b[P::b_map(seg, n_tile, grp, ep)], &full_bar[stage],
                              P::b_col(seg, n_tile, grp, ep), kb * GEMM_BK, pc);
              } else {
                tma_load_3d(sb + pc * P::BN * 128, &maps.b[P::b_map(seg, n_tile, 0, ep)], &full_bar[stage], kb * GEMM_BK,
                            P::b_col(seg, n_tile, 0, ep), pc);
              }
            }
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
      constexpr uint32_t idesc = umma_idesc_bf16(GEMM_BM, P::BN) | (P::B_MN ? UMMA_B_MN : 0u);
      using T = Terms<P::PA, P::PB>;
      int stage = 0;
      uint32_t phase = 0, it = 0;
      bool alive = true;
      for (long long tile = blockIdx.x; tile < total && alive; tile += gridDim.x, ++it) {
        const int split = static_cast<int>(tile % g.splits);
        const uint32_t buf = it % NBUF, buf_phase = (it / NBUF) & 1;
        if (!mbar_wait(&acc_empty[buf], buf_phase ^ 1, g.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        for (int seg = 0; seg < P::NSEG && alive; ++seg) {
          const uint32_t d_seg = tmem_base + buf * ACC + seg * SEG;
          const int per = (g.kb[seg] + g.splits - 1) / g.splits;
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
              const uint64_t adesc = umma_desc_kmajor(sa + T::a(t) * GEMM_A_BYTES, 128);
              const uint64_t bdesc = P::B_MN ? umma_desc_mnmajor(sb + T::b(t) * P::BN * 128, 8192)
                                             : umma_desc_kmajor(sb + T::b(t) * P::BN * 128, 128);
              const bool lead = t == T::N - 1;
              const uint32_t d_tmem = d_seg + (lead ? (kb - k0) % P::NMAIN : P::NMAIN) * P::BN;
              const int fresh = lead ? kb - k0 < P::NMAIN : (kb == k0 && t == 0);  // first product into it
#pragma unroll
              for (int k = 0; k < GEMM_BK / 16; ++k)
                umma_bf16_ss(d_tmem, umma_desc_advance(adesc, k * 32), umma_desc_advance(bdesc, P::B_MN ? k * 2048 : k * 32),
                             idesc, !(fresh && k == 0));
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
    const int quarter = warp & 3, half = (warp - 4) >> 2;
    uint32_t it = 0;
    for (long long tile = blockIdx.x; tile < total; tile += gridDim.x, ++it) {
      const int split = static_cast<int>(tile % g.splits);
      const int n_tile = static_cast<int>((tile / g.splits) % g.n_tiles);
      const int m_tile = static_cast<int>(tile / g.splits / g.n_tiles);
      const uint32_t buf = it % NBUF, buf_phase = (it / NBUF) & 1;
      if (!mbar_wait(&acc_full[buf], buf_phase, g.status, ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      const int per = (g.kb[0] + g.splits - 1) / g.splits;
      const Accum<P> acc = {tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * ACC,
                            min(g.kb[0], (split + 1) * per) - split * per};
      P::epilogue(ep, m_tile, n_tile, split, acc, quarter, half, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
  }

  if (*reinterpret_cast<volatile int*>(g.status) != ST_OK)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
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
  const unsigned grid = static_cast<unsigned>(total < sm_count() ? total : sm_count());
  return launch(piece_gemm_kernel<P>, dim3(grid), dim3(GEMM_THREADS), gemm_smem_bytes<P>(), stream, pdl, maps, g, ep);
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
// Weights as stored, [k][n] with row pitch `pitch` (a multiple of 8), read as MN-major tiles.
inline int gemm_map_mnmajor(CUtensorMap* out, const void* base, int k, int n, long long pitch) {
  const uint64_t dims[3] = {static_cast<uint64_t>(n), static_cast<uint64_t>(k), 1};
  const uint64_t str[2] = {static_cast<uint64_t>(pitch) * 2, static_cast<uint64_t>(pitch) * k * 2};
  const uint32_t box[3] = {64, GEMM_BK, 1};
  return make_tmap(out, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
}

}  // namespace b200
