// Attention core in float32 arithmetic on the tensor cores: the triangle attention of a float32
// trunk and of bf16 trunks of any head shape (rows i of the pair tensor share the bias), and
// the single track's token attention (one row, 16 heads of width 24).
//
//   S = (q . k) * scale + mask_bias + bias        o = softmax(S) . v
//
// q, k, v arrive as bf16 pieces (gemm.cuh): three when they are float32, one when the trunk is bf16,
// which has a kernel of its own below. The probabilities are split into three pieces by the thread that
// computes them, so P.V is as exact as a float32 product. The piece products of one result are issued
// smallest first into one float32 accumulator, so that only the leading one is summed at full
// magnitude. Everything in between is float32 as in the reference (_attention_block,
// src/foldjax/models/boltz2/models/triangle/triangle_attention.py:428-455;
// _attention_qblock, primitives/attention.py:124-140): softmax in float32. With float32 operands
// the running numerator stays in registers (P.V of a step starts from zero and is added by the
// thread, which also makes the rescale a register fma).
//
// One CTA per SM, persistent; an item is (head, NWG rows, 128 queries), or with one row (head,
// NWG tiles of 128 queries), walked in steps of 64 keys, the last one of as many columns as it needs:
//   warp 0      TMA producer       warp 1   S issuer       warps 2, 3   P.V issuers, one for each row or tile
//   warpgroups  softmax, one thread per query
// Bound of the float32 kernel: two softmax warpgroups fill 41 % of the issue slots (counters, 512 tokens, 4 heads x
// 32, 565 us; a score costs about 2 instructions of exponential, 3.5 of split and 4 others, most of them packed two to an
// instruction; with 4.5 of split it was 41 % and 575); the rest is products (1300 clocks of the tensor pipe for a row's step) and loads, 80 KiB a step and SM.
#include <climits>
#include <type_traits>

#include "att_split.cuh"
#include "gemm.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int KT = 64;

// NWG: softmax warpgroups, each with a row, or (TOKEN) with 128 queries, of its own.
template <int HDP, bool TOKEN, int NWG_>
struct Cfg {
  static constexpr int NWG = NWG_;
  static constexpr int KV = TOKEN ? 1 : NWG;  // rows whose keys a step loads
  static constexpr int NB = TOKEN ? NWG : 1;  // bias tiles of a step
  static constexpr int STAGES = 2;
  static constexpr int THREADS = 128 + NWG * 128;
  static constexpr int Q_BYTES = 128 * HDP * 2, K_BYTES = KT * HDP * 2, V_BYTES = HDP * 128;
  static constexpr int BIAS_BYTES = 128 * KT * 4;
  static constexpr uint32_t TM_S = 0, TM_P = 64, TM_O = TM_P + 96, TM_WG = TM_O + HDP;
  static_assert(NWG * TM_WG <= 512, "tensor memory budget");
  static constexpr uint32_t STAGE_TX = KV * 3 * (K_BYTES + V_BYTES) + NB * BIAS_BYTES + KV * KT * 4;
};

template <int HDP, bool TOKEN, int NWG>
struct Smem {
  using C = Cfg<HDP, TOKEN, NWG>;
  uint8_t q[C::NWG][3][C::Q_BYTES];
  uint8_t k[C::STAGES][C::KV][3][C::K_BYTES];
  uint8_t v[C::STAGES][C::KV][3][C::V_BYTES];
  uint8_t bias[C::STAGES][C::NB][C::BIAS_BYTES];  // two boxes of 32 keys, [128 queries][32 floats]
  alignas(128) float mb[C::STAGES][C::KV][KT];
  uint64_t q_full, q_empty, st_full[C::STAGES], st_empty[C::STAGES], s_full[C::NWG], s_free[C::NWG], p_full[C::NWG],
      pv_done[C::NWG];
  uint32_t tmem_base;
};

struct Maps {
  CUtensorMap q, k, v, b, m;
};

struct Params {
  int n_i, n, heads, head_dim;
  int groups, tiles_j, steps;
  uint32_t total_items;
  float scale;
  void* o;                   // [rows][n][heads * head_dim], float32, or bf16 with bf16 operands
  const float* gate;         // one row: the output is o * gate as pieces
  __nv_bfloat16* pieces;     // [3][n][heads * head_dim]
  int* status;
};

// e^(s - m) for two scores, m at least their maximum so far. The difference comes first, so the
// error of 2^t is about 2^-23 |t| of a weight 2^-|t|: never above 2^-24 of the largest weight.
__device__ __forceinline__ float2 exp_below(float2 s, float2 minus_m) {
  const float2 t = __fmul2_rn(__fadd2_rn(s, minus_m), make_float2(1.44269504f, 1.44269504f));
  return make_float2(fast_exp2(t.x), fast_exp2(t.y));
}

template <int HDP, bool TOKEN, int NWG, int LAST>
__global__ void __launch_bounds__(Cfg<HDP, TOKEN, NWG>::THREADS, 1)
att_split_kernel(const __grid_constant__ Maps tm, const Params p) {
  using C = Cfg<HDP, TOKEN, NWG>;
  using TQ = Terms<3, 3>;  // q . k
  using TP = Terms<3, 3>;  // P . v
  constexpr int STAGES = C::STAGES;
  static_assert(sizeof(Smem<HDP, TOKEN, NWG>) <= 232448, "shared memory budget");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem<HDP, TOKEN, NWG>& sm = *reinterpret_cast<Smem<HDP, TOKEN, NWG>*>(smem_raw);
  // (through a shuffle, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, ST_OK, 900);
    return;
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm.q);
    tma_prefetch_desc(&tm.k);
    tma_prefetch_desc(&tm.v);
    tma_prefetch_desc(&tm.b);
    mbar_init(&sm.q_full, 1);
    mbar_init(&sm.q_empty, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm.st_full[s], 1);
      mbar_init(&sm.st_empty[s], NWG + NWG * 4);
    }
    for (int g = 0; g < NWG; ++g) {
      mbar_init(&sm.s_full[g], 1);
      mbar_init(&sm.s_free[g], 128);
      mbar_init(&sm.p_full[g], 128);
      mbar_init(&sm.pv_done[g], 1);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem_base = sm.tmem_base;
  const uint32_t items_per_head = p.groups * p.tiles_j;
  // item -> head, batch item, row inside it and first query of warpgroup 0; the others follow at
  // successive rows, or (one row) at successive tiles of 128 queries
  auto locate = [&](uint32_t item, int& b, int& h, int& i, int& j0) {
    const uint32_t bh = item / items_per_head, rem = item - bh * items_per_head;
    b = bh / p.heads;
    h = bh - b * p.heads;
    const uint32_t grp = rem / p.tiles_j, tile = rem - grp * p.tiles_j;
    i = grp * NWG;  // (one group of rows in the one-row form)
    j0 = tile * (TOKEN ? NWG * 128 : 128);
  };

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0, item_it = 0;
      bool alive = true;
      for (uint32_t item = blockIdx.x; item < p.total_items && alive; item += gridDim.x, ++item_it) {
        if (!mbar_wait(&sm.q_empty, (item_it & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
        mbar_expect_tx(&sm.q_full, NWG * 3 * C::Q_BYTES);
        int b, h, i, j0;
        locate(item, b, h, i, j0);
        const int row = b * p.n_i + i;
        for (int g = 0; g < NWG; ++g)
          for (int pc = 0; pc < 3; ++pc)
            tma_load_5d(sm.q[g][pc], &tm.q, &sm.q_full, 0, h, TOKEN ? j0 + g * 128 : j0, TOKEN ? row : row + g, pc);
        for (int t = 0; t < p.steps; ++t) {
          if (!mbar_wait(&sm.st_empty[stage], phase ^ 1, p.status, ST_TIMEOUT_PRODUCER)) {
            alive = false;
            break;
          }
          const int k0 = t * KT;
          mbar_expect_tx(&sm.st_full[stage], C::STAGE_TX);
#pragma unroll 1
          for (int g = 0; g < C::KV; ++g) {
#pragma unroll 1
            for (int pc = 0; pc < 3; ++pc) {
              tma_load_5d(sm.k[stage][g][pc], &tm.k, &sm.st_full[stage], 0, h, k0, row + g, pc);
              tma_load_5d(sm.v[stage][g][pc], &tm.v, &sm.st_full[stage], k0, 0, h, row + g, pc);
            }
            tma_load_2d(sm.mb[stage][g], &tm.m, &sm.st_full[stage], k0, row + g);
          }
          for (int g = 0; g < C::NB; ++g) {
            for (int half = 0; half < 2; ++half)
              tma_load_4d(sm.bias[stage][g] + half * 16384, &tm.b, &sm.st_full[stage], k0 + half * 32, j0 + g * 128, h, b);
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // In the issuers all lanes walk the loops and wait, and one of them issues; none leaves early: one whose wait has run out
    // stops waiting and issuing and walks on. Joins as in triatt_core.cu.
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0, item_it = 0, g = 0;
    bool alive = true;
    for (uint32_t item = blockIdx.x; item < p.total_items; item += gridDim.x, ++item_it) {
      alive = alive && mbar_wait(&sm.q_full, item_it & 1, p.status, ST_TIMEOUT_MMA);
      for (int t = 0; t < p.steps; ++t, ++g) {
        alive = alive && mbar_wait(&sm.st_full[stage], phase, p.status, ST_TIMEOUT_MMA);
        const uint32_t idesc = umma_idesc_bf16(128, LAST < KT && t + 1 == p.steps ? LAST : KT);
#pragma unroll
        for (int wg = 0; wg < NWG; ++wg) {
          alive = alive && mbar_wait(&sm.s_free[wg], (g & 1) ^ 1, p.status, ST_TIMEOUT_MMA);
          __syncwarp();
          tc_fence_after();
          const uint32_t d = tmem_base + wg * C::TM_WG + C::TM_S;
          if (leader && alive) {
#pragma unroll
            for (int term = 0; term < TQ::N; ++term) {
              const uint64_t adesc = umma_desc_kmajor(smem_u32(sm.q[wg][TQ::a(term)]), HDP * 2);
              const uint64_t bdesc = umma_desc_kmajor(smem_u32(sm.k[stage][TOKEN ? 0 : wg][TQ::b(term)]), HDP * 2);
#pragma unroll
              for (int kk = 0; kk < HDP / 16; ++kk)
                umma_bf16_ss(d, umma_desc_advance(adesc, kk * 32), umma_desc_advance(bdesc, kk * 32), idesc,
                             (term | kk) != 0);
            }
            umma_commit(&sm.s_full[wg]);
          }
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (leader && alive) umma_commit(&sm.q_empty);
    }
  } else if (warp < 2 + NWG) {  // P.V of a row each
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, HDP);
    const int wg = warp - 2;
    int stage = 0;
    uint32_t phase = 0, g = 0;
    bool alive = true;
    for (uint32_t item = blockIdx.x; item < p.total_items; item += gridDim.x) {
      for (int t = 0; t < p.steps; ++t, ++g) {
        alive = alive && mbar_wait(&sm.st_full[stage], phase, p.status, ST_TIMEOUT_MMA);
        alive = alive && mbar_wait(&sm.p_full[wg], g & 1, p.status, ST_TIMEOUT_MMA);
        __syncwarp();
        tc_fence_after();
        const int cols = LAST < KT && t + 1 == p.steps ? LAST : KT;
        const uint32_t base = tmem_base + wg * C::TM_WG;
        const uint32_t vbase = smem_u32(sm.v[stage][TOKEN ? 0 : wg][0]);
        if (leader && alive) {
#pragma unroll
          for (int term = 0; term < TP::N; ++term) {
            const uint64_t vdesc = umma_desc_kmajor(vbase + TP::b(term) * C::V_BYTES, 128);
#pragma unroll
            for (int kk = 0; kk < KT / 16; ++kk)
              if (kk * 16 < LAST || kk * 16 < cols)
                umma_bf16_ts(base + C::TM_O, base + C::TM_P + TP::a(term) * 32 + kk * 8, umma_desc_advance(vdesc, kk * 32),
                             idesc, (term | kk) != 0);
          }
          umma_commit(&sm.pv_done[wg]);
          umma_commit(&sm.st_empty[stage]);
        }
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp >= 4) {
    const int wg = (warp - 4) >> 2, quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t t_wg = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + wg * C::TM_WG;
    int stage = 0;
    uint32_t phase = 0, g = 0;
    bool alive = true;
    for (uint32_t item = blockIdx.x; item < p.total_items && alive; item += gridDim.x) {
      float m_run = -INFINITY, l_run = 0.f, alpha = 0.f;
      float o[HDP];
#pragma unroll
      for (int d = 0; d < HDP; ++d) o[d] = 0.f;
      auto take_pv = [&] {  // o = o * (rescale of the step P.V belongs to) + P.V
#pragma unroll
        for (int part = 0; part < HDP / 16; ++part) {
          uint32_t r[16];
          tmem_ld16(t_wg + C::TM_O + part * 16, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float& acc = o[part * 16 + e];
            acc = fmaf(acc, alpha, __uint_as_float(r[e]));
          }
        }
      };
      // A step of COLS keys; what the last one leaves out of 64 are keys that do not exist.
      auto step = [&](auto width, int t) -> bool {
        constexpr int COLS = decltype(width)::value;
        // (votes: each lane polls for itself, TMEM accesses take the whole warp, and all or none of it leave)
        alive = mbar_wait(&sm.st_full[stage], phase, p.status, ST_TIMEOUT_SOFTMAX) &&
                mbar_wait(&sm.s_full[wg], g & 1, p.status, ST_TIMEOUT_SOFTMAX);
        if (!__all_sync(0xffffffffu, alive)) {
          alive = false;
          return false;
        }
        tc_fence_after();
        float2 s[COLS / 2];
        {
          uint32_t r[COLS];
          if constexpr (COLS >= 32) tmem_ld32(t_wg + C::TM_S, reinterpret_cast<uint32_t(&)[32]>(r));
          if constexpr (COLS == 64) tmem_ld32(t_wg + C::TM_S + 32, reinterpret_cast<uint32_t(&)[32]>(r[32]));
          if constexpr (COLS % 32 == 16) tmem_ld16(t_wg + C::TM_S + COLS - 16, reinterpret_cast<uint32_t(&)[16]>(r[COLS - 16]));
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < COLS / 2; ++e) s[e] = make_float2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
        }
        tc_fence_before();
        mbar_arrive(&sm.s_free[wg]);
        const float* mrow = sm.mb[stage][TOKEN ? 0 : wg];
        const bool masked = __any_sync(0xffffffffu, ((COLS >= 32 || lane < COLS) && mrow[lane] != 0.f) ||
                                                         ((COLS == 64 || lane + 32 < COLS) && mrow[lane + 32] != 0.f));
        // the reference's order of the two sums
        const uint8_t* brow = sm.bias[stage][TOKEN ? wg : 0];
#pragma unroll
        for (int c = 0; c < COLS / 4; ++c) {
          const float4 b4 = *reinterpret_cast<const float4*>(brow + (c >> 3) * 16384 + sw128_offset(row, c & 7));
          const float2 b2[2] = {make_float2(b4.x, b4.y), make_float2(b4.z, b4.w)};
          float2 m2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          if ((c & 1) == 1) asm volatile("" ::: "memory");  // keep the loads from piling up in registers
          if (masked) {
            const float4 m4 = *reinterpret_cast<const float4*>(mrow + 4 * c);
            m2[0] = make_float2(m4.x, m4.y);
            m2[1] = make_float2(m4.z, m4.w);
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            float2& x = s[2 * c + u];
            x = TOKEN ? __fadd2_rn(__ffma2_rn(x, make_float2(p.scale, p.scale), b2[u]), m2[u])
                      : __fadd2_rn(__fadd2_rn(x, m2[u]), b2[u]);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.st_empty[stage]);
        float mxa = m_run, mxb = s[0].x;
#pragma unroll
        for (int e = 0; e < COLS / 2; e += 2) {
          mxa = fmax3(mxa, s[e].x, s[e].y);
          mxb = fmax3(mxb, s[e + 1].x, s[e + 1].y);
        }
        const float mx = fmaxf(mxa, mxb);  // (with the running maximum in it)
        const float alpha_new = fast_exp2((m_run - mx) * 1.44269504f);  // 0 on the first step
        m_run = mx;
        float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int e = 0; e < COLS / 2; ++e) {
          s[e] = exp_below(s[e], make_float2(-mx, -mx));
          l2[e & 1] = __fadd2_rn(l2[e & 1], s[e]);
        }
        l_run = fmaf(l_run, alpha_new, (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y));
        // the previous step's P.V: its result is taken, then P may be overwritten
        alive = mbar_wait(&sm.pv_done[wg], (g & 1) ^ 1, p.status, ST_TIMEOUT_SOFTMAX);
        if (!__all_sync(0xffffffffu, alive)) {
          alive = false;
          return false;
        }
        tc_fence_after();
        if (t > 0) take_pv();
        alpha = alpha_new;
#pragma unroll
        for (int oct = 0; oct < COLS / 16; ++oct) {  // 16 keys at a time: few live registers
          uint32_t pc[3][8];
#pragma unroll
          for (int e = 0; e < 8; ++e) split3x2(s[oct * 8 + e].x, s[oct * 8 + e].y, pc[0][e], pc[1][e], pc[2][e]);
#pragma unroll
          for (int q = 0; q < 3; ++q) tmem_st8(t_wg + C::TM_P + q * 32 + oct * 8, pc[q]);
        }
        tmem_st_wait();
        tc_fence_before();
        mbar_arrive(&sm.p_full[wg]);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
        return true;
      };
      const int whole = LAST < KT ? p.steps - 1 : p.steps;
      for (int t = 0; t < whole; ++t, ++g)
        if (!step(std::integral_constant<int, KT>{}, t)) break;
      if constexpr (LAST < KT) {
        if (alive) step(std::integral_constant<int, LAST>{}, whole);
        ++g;
      }
      if (!alive) break;
      if (!__all_sync(0xffffffffu, mbar_wait(&sm.pv_done[wg], (g & 1) ^ 1, p.status, ST_TIMEOUT_SOFTMAX))) break;
      tc_fence_after();
      take_pv();
      int b, h, i, j0;
      locate(item, b, h, i, j0);
      if (TOKEN)
        j0 += wg * 128;
      else
        i += wg;
      const int j = j0 + row;
      const bool live = i < p.n_i && j < p.n;
      const long long off = ((static_cast<long long>(b * p.n_i + i) * p.n + j) * p.heads + h) * p.head_dim;
      const float inv = 1.0f / l_run;
      tc_fence_before();
      if constexpr (TOKEN) {
        const long long plane = static_cast<long long>(p.n) * p.heads * p.head_dim;
#pragma unroll
        for (int d = 0; d < HDP; d += 8) {
          if (!live || d >= p.head_dim) break;
          uint32_t w[3][4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            split3x2(o[d + 2 * e] * inv * p.gate[off + d + 2 * e], o[d + 2 * e + 1] * inv * p.gate[off + d + 2 * e + 1], w[0][e],
                     w[1][e], w[2][e]);
#pragma unroll
          for (int q = 0; q < 3; ++q)
            *reinterpret_cast<uint4*>(p.pieces + q * plane + off + d) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
        }
      } else {
#pragma unroll
        for (int d = 0; d < HDP; d += 8)
          if (live && d < p.head_dim) {  // (a multiple of 8)
            uint32_t w[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(o[d + e] * inv);
            store_sector(static_cast<float*>(p.o) + off + d, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
          }
      }
    }
  }

  if (*reinterpret_cast<volatile int*>(p.status) != ST_OK)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// Calls go with the columns of an item's last step as a constant: 16, 32, 48 or 64, whichever hold the keys that are left.
// (Templates of 200 tokens 610 -> 590 us, 150-token refiner 499 -> 487, 200-token float32 stack 644 -> 642, blocks of 136 and
// 203 tokens, single track only, 198.7 -> 197.2 and 262.7 -> 261.6; the same bits.)
// STEPS48: most steps of an item whose last one takes 48 columns instead of 64. Us of a core with 64 and with 48, 100 / 170 / 240 tokens:
// 4 bf16 heads x 16 9.0 / 27.4 / 41.5 and 8.7 / 26.2 / 39.6, 12 x 32 22.1 / 60.3 / 105 and 21.4 / 57.3 / 98.6; float32 4 x 32 26.6 /
// 57.3 / 96.8 and 26.0 / 58.4 / 98.4; but bf16 4 x 64 20.7 / 44.7 / 70.4 and 21.0 / 45.0 / 72.6, float32 2 x 64 24.8 / 55.5 / 89.9 and
// 25.3 / 56.3 / 90.4, single track 12.9 / 15.7 / 17.1 and 13.1 / 15.8 / 17.1: none there.
template <int STEPS48, class F>
int with_last_columns(const Params& p, const F& go) {
  switch (round_up(p.n - KT * (p.steps - 1), 16)) {
    case 16: return go(std::integral_constant<int, 16>{});
    case 32: return go(std::integral_constant<int, 32>{});
    case 48:
      if constexpr (STEPS48 > 0)
        if (p.steps <= STEPS48) return go(std::integral_constant<int, 48>{});
  }
  return go(std::integral_constant<int, KT>{});
}

template <int HDP, bool TOKEN, int NWG>
int launch_cfg(const Maps& tm, Params p, bool pdl, cudaStream_t stream) {
  using C = Cfg<HDP, TOKEN, NWG>;
  const int tiles = (p.n + 127) / 128;
  p.groups = TOKEN ? 1 : (p.n_i + C::NWG - 1) / C::NWG;
  p.tiles_j = TOKEN ? (tiles + C::NWG - 1) / C::NWG : tiles;
  const long long items = static_cast<long long>(p.total_items) * p.groups * p.tiles_j;
  B200_REQUIRE(items < (1ll << 32) - 1024, B200TRI_ERR_UNSUPPORTED, "float32 attention: too many tiles");
  p.total_items = static_cast<uint32_t>(items);
  return with_last_columns<HDP == 32 && !TOKEN ? 2 : 0>(p, [&](auto last) {
    const auto kernel = att_split_kernel<HDP, TOKEN, NWG, decltype(last)::value>;
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), (int)sizeof(Smem<HDP, TOKEN, NWG>));
    if (rc) return rc;
    const unsigned sms = sm_count(), grid = p.total_items < sms ? p.total_items : sms;
    return launch(kernel, dim3(grid), dim3(C::THREADS), sizeof(Smem<HDP, TOKEN, NWG>), stream, pdl, tm, p);
  });
}


// ------------------------------------------------------------------------- bf16 operands
// The same core where q, k, v and the bias are bf16. The bias is added by the tensor core, as in
// triatt_core.cu (S = bias . I + q . k), the numerator accumulates in TMEM and is rescaled only when
// the maximum grew by more than RESCALE, and the probabilities overwrite the scores they came from, so
// that four softmax warpgroups fit (128 columns each).
//   warp 0       TMA producer            warps 1, 2   P.V issuers, each of half of the rows (three rows: one)
//   warp 3       issuer of all scores    warpgroups   softmax, one thread per query
// A row's next scores go to columns that P.V of this step reads. Products of other shapes into other accumulators
// have no order that is promised, whoever issued them, so warp 3 waits until P.V is through; s_full then tells the
// softmax that both are. A warp of its own, because one that issued P.V too kept its other rows' P.V waiting
// (attention of 320 tokens, 4 heads x 32, 155 us; 150 with both issued back to back and no wait; 148 so).
// The softmax offset is an integer in log2 units (one fma per pair of exponentials, exact
// powers of two to rescale by) except where scores are so large that integers are no finer than they are.
//
// Bound: a row's step is a chain of softmax (1.2 us with the other rows' warps beside it, 8 instructions a
// score) and products (18 of them, 0.35 us, and the trips between the warps), and the rows in flight hide
// each other's. Three rows, P.V issued by one warp, padded heads of 16, rounded pieces and pairs unpacked from them
// took 695 us for the four updates of four 200-token templates, 1 178 for those of a 256-token refiner, 112 and 247 for
// attention of 200 and 320 tokens with 4 heads x 64; 615, 1 130, 105 and 219 so. It issues in 69 % of its slots with 65 % of
// the MUFU unit busy (counters, 4 x 400 tokens, 4 heads x 16).
// HDP: a head's width in the products, rounded up to 16, 32 or 64. Heads of 16 as 32 pay for a product of
// zeros a step and twice the columns in P.V, and read back twice the result: 2.3 % of the templates' time (the same bits).
// Measured and not better: an issuer per row, rows started a fraction of a step apart, P as two tf32 pieces
// against V as float32, ending an item with its rows' last kept key (the flags cost the issuers 4 %, which
// only paddings of a whole step pay back), the difference of two bf16 by a subtraction.
template <int HDP, int NWG>
struct BfCfg {
  static constexpr int STAGES = 3, QBUF = 2, THREADS = 128 + NWG * 128;
  static constexpr int ISSUERS = NWG == 3 ? 1 : 2, ROWS = NWG / ISSUERS;  // rows of an issuer
  // Registers of the control and of the softmax warpgroups, out of those the block is launched with:
  // 512 x 128 = 128 x 56 + 384 x 152, 640 x 96 = 128 x 32 + 512 x 112 (two rows have enough as they are)
  static constexpr int CONTROL_REGS = NWG == 4 ? 32 : 56, SOFTMAX_REGS = NWG == 4 ? 112 : 152;
  static constexpr int Q_BYTES = 128 * HDP * 2, K_BYTES = KT * HDP * 2, V_BYTES = HDP * 128, BIAS_BYTES = 128 * KT * 2;
  static constexpr uint32_t TM_P = 0, TM_O = 96, TM_WG = HDP <= 32 ? 128 : TM_O + HDP;  // P (three pieces) over S (64 columns)
  static_assert(NWG * TM_WG <= 512, "tensor memory budget");
  static constexpr uint32_t STAGE_TX = NWG * (K_BYTES + V_BYTES + KT * 4) + BIAS_BYTES;
};

template <int HDP, int NWG>
struct BfSmem {
  using C = BfCfg<HDP, NWG>;
  uint8_t q[C::QBUF][NWG][C::Q_BYTES];
  uint8_t k[C::STAGES][NWG][C::K_BYTES];
  uint8_t v[C::STAGES][NWG][C::V_BYTES];
  uint8_t bias[C::STAGES][C::BIAS_BYTES];  // [128 queries][64 keys]
  uint8_t ident[KT * 128];                 // 64 x 64 bf16 identity
  alignas(128) float mb[C::STAGES][NWG][KT];
  uint64_t q_full[C::QBUF], q_empty[C::QBUF], st_full[C::STAGES], st_empty[C::STAGES], s_full[NWG], p_full[NWG], pv_done[NWG];
  uint32_t tmem_base;
};

// The numerator is rescaled when a maximum exceeds the one that gave the offset by so much. An offset in whole log2
// units lies up to half a unit below its maximum, so weights stay below e^5.5 * 2^0.5 = 346.
constexpr float RESCALE = 5.5f;
constexpr float LOG2E = 1.44269504f;
constexpr float INTEGER_OFFSETS = 8388608.0f;  // 2^23: floats beyond are integers themselves

// hi + mid + lo = v exactly, and all three go into P.V: bf16 is the upper half of a float, and its 8 bits leave 16 and
// then 8 of the 24. Cut off instead of rounded, as exact and a byte permutation for two instead of a conversion:
// templates 634 -> 623 us, 4 x 320 tokens 445 -> 434; error against float64 over 40 inputs within 1e-5 of itself either way,
// 7e-7 on average.
__device__ __forceinline__ uint32_t upper_halves(float2 v) {
  return __byte_perm(__float_as_uint(v.x), __float_as_uint(v.y), 0x7632);
}
__device__ __forceinline__ void split3n2(float2 v, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = upper_halves(v);
  const float2 r = less_bf16x2(v, hi);
  mid = upper_halves(r);
  lo = upper_halves(less_bf16x2(r, mid));
}

template <int HDP, int NWG, int LAST>
__global__ void __launch_bounds__(BfCfg<HDP, NWG>::THREADS, 1)
att_bf16_kernel(const __grid_constant__ Maps tm, const Params p) {
  using C = BfCfg<HDP, NWG>;
  using TP = Terms<3, 1>;  // P . v
  constexpr int STAGES = C::STAGES;
  static_assert(sizeof(BfSmem<HDP, NWG>) <= 232448, "shared memory budget");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  BfSmem<HDP, NWG>& sm = *reinterpret_cast<BfSmem<HDP, NWG>*>(smem_raw);
  // (through a shuffle, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, ST_OK, 900);
    return;
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm.q);
    tma_prefetch_desc(&tm.k);
    tma_prefetch_desc(&tm.v);
    tma_prefetch_desc(&tm.b);
    for (int b = 0; b < C::QBUF; ++b) {
      mbar_init(&sm.q_full[b], 1);
      mbar_init(&sm.q_empty[b], 1);
    }
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm.st_full[s], 1);
      mbar_init(&sm.st_empty[s], C::ISSUERS + NWG * 4);
    }
    for (int g = 0; g < NWG; ++g) {
      mbar_init(&sm.s_full[g], 1);
      mbar_init(&sm.p_full[g], 4);
      mbar_init(&sm.pv_done[g], 1);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  for (int idx = threadIdx.x; idx < KT * 32; idx += C::THREADS) {  // the identity, K-major under the 128-byte swizzle
    const int r = idx / 32, w = idx % 32;
    const int e0 = ((w >> 2) ^ (r & 7)) * 8 + (w & 3) * 2;  // logical element of the word's low half
    reinterpret_cast<uint32_t*>(sm.ident)[idx] = e0 == r ? 0x00003F80u : e0 + 1 == r ? 0x3F800000u : 0u;
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();
  pdl_trigger();
  const uint32_t tmem_base = sm.tmem_base;
  const uint32_t items_per_head = p.groups * p.tiles_j;
  // item -> head, batch item, first row inside it and first query
  auto locate = [&](uint32_t item, int& b, int& h, int& i, int& j0) {
    const uint32_t bh = item / items_per_head, rem = item - bh * items_per_head;
    b = bh / p.heads;
    h = bh - b * p.heads;
    const uint32_t grp = rem / p.tiles_j;
    i = grp * NWG;
    j0 = (rem - grp * p.tiles_j) * 128;
  };

  // In warps 0 to 3 all lanes walk the loops and wait, and one of them issues; none leaves early: one whose
  // wait has run out stops waiting and issuing and walks on. Joins as in triatt_core.cu.
  if (warp < 4) {
    if (NWG > 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::CONTROL_REGS));
    if (warp == 0) {
      const bool leader = elect_one();
      int stage = 0;
      uint32_t phase = 0, item_it = 0;
      bool alive = true;
      for (uint32_t item = blockIdx.x; item < p.total_items; item += gridDim.x, ++item_it) {
        int b, h, i, j0;
        locate(item, b, h, i, j0);
        const int row = b * p.n_i + i;
        const uint32_t qb = item_it % C::QBUF;
        alive = alive && mbar_wait(&sm.q_empty[qb], ((item_it / C::QBUF) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER);
        __syncwarp();
        if (leader && alive) {
          mbar_expect_tx(&sm.q_full[qb], NWG * C::Q_BYTES);
          for (int g = 0; g < NWG; ++g) tma_load_5d(sm.q[qb][g], &tm.q, &sm.q_full[qb], 0, h, j0, row + g, 0);
        }
        for (int t = 0; t < p.steps; ++t) {
          alive = alive && mbar_wait(&sm.st_empty[stage], phase ^ 1, p.status, ST_TIMEOUT_PRODUCER);
          __syncwarp();
          const int k0 = t * KT;
          if (leader && alive) {
            mbar_expect_tx(&sm.st_full[stage], C::STAGE_TX);
            tma_load_4d(sm.bias[stage], &tm.b, &sm.st_full[stage], k0, j0, h, b);
            for (int g = 0; g < NWG; ++g) {
              tma_load_5d(sm.k[stage][g], &tm.k, &sm.st_full[stage], 0, h, k0, row + g, 0);
              tma_load_2d(sm.mb[stage][g], &tm.m, &sm.st_full[stage], k0, row + g);
              tma_load_5d(sm.v[stage][g], &tm.v, &sm.st_full[stage], k0, 0, h, row + g, 0);
            }
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    } else if (warp <= C::ISSUERS) {
      const bool leader = elect_one();
      const int r0 = (warp - 1) * C::ROWS;
      constexpr uint32_t idesc = umma_idesc_bf16(128, HDP);
      int stage = 0;
      uint32_t phase = 0, g = 0;  // g: steps so far
      bool alive = true;
      for (uint32_t item = blockIdx.x; item < p.total_items; item += gridDim.x) {
        for (int t = 0; t < p.steps; ++t, ++g) {
          // (already complete when P arrives; observed here so that this thread's products are ordered after the
          // TMA writes of V)
          alive = alive && mbar_wait(&sm.st_full[stage], phase, p.status, ST_TIMEOUT_MMA);
          const int cols = LAST < KT && t + 1 == p.steps ? LAST : KT;
#pragma unroll 1
          for (int u = 0; u < C::ROWS; ++u) {
            const int wg = r0 + u;
            alive = alive && mbar_wait(&sm.p_full[wg], g & 1, p.status, ST_TIMEOUT_MMA);
            __syncwarp();
            tc_fence_after();
            const uint32_t base = tmem_base + wg * C::TM_WG;
            const uint64_t vdesc = umma_desc_kmajor(smem_u32(sm.v[stage][wg]), 128);
            if (leader && alive) {
#pragma unroll
              for (int term = 0; term < TP::N; ++term)
#pragma unroll
                for (int kk = 0; kk < KT / 16; ++kk)
                  if (kk * 16 < LAST || kk * 16 < cols)
                    umma_bf16_ts(base + C::TM_O, base + C::TM_P + TP::a(term) * 32 + kk * 8, umma_desc_advance(vdesc, kk * 32),
                                 idesc, t > 0 || (term | kk) != 0);
              umma_commit(&sm.pv_done[wg]);
            }
          }
          if (leader && alive) umma_commit(&sm.st_empty[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    } else if (warp == 3) {
      const bool leader = elect_one();
      const uint64_t identdesc = umma_desc_kmajor(smem_u32(sm.ident), 128);
      int stage = 0;
      uint32_t phase = 0, item_it = 0, g = 0;
      bool alive = true;
      for (uint32_t item = blockIdx.x; item < p.total_items; item += gridDim.x, ++item_it) {
        const uint32_t qb = item_it % C::QBUF;
        alive = alive && mbar_wait(&sm.q_full[qb], (item_it / C::QBUF) & 1, p.status, ST_TIMEOUT_MMA);
        for (int t = 0; t < p.steps; ++t, ++g) {
          alive = alive && mbar_wait(&sm.st_full[stage], phase, p.status, ST_TIMEOUT_MMA);
          const int cols = LAST < KT && t + 1 == p.steps ? LAST : KT;
          const uint32_t idesc = umma_idesc_bf16(128, cols);
          const uint64_t biasdesc = umma_desc_kmajor(smem_u32(sm.bias[stage]), 128);
#pragma unroll 1
          for (int wg = 0; wg < NWG; ++wg) {
            // the scores' columns are free once the products that read P in them are through
            alive = alive && mbar_wait(&sm.pv_done[wg], (g & 1) ^ 1, p.status, ST_TIMEOUT_MMA);
            __syncwarp();
            tc_fence_after();
            const uint32_t d = tmem_base + wg * C::TM_WG;
            const uint64_t adesc = umma_desc_kmajor(smem_u32(sm.q[qb][wg]), HDP * 2);
            const uint64_t bdesc = umma_desc_kmajor(smem_u32(sm.k[stage][wg]), HDP * 2);
            if (leader && alive) {
#pragma unroll
              for (int kk = 0; kk < KT / 16; ++kk)
                if (kk * 16 < LAST || kk * 16 < cols)
                  umma_bf16_ss(d, umma_desc_advance(biasdesc, kk * 32), umma_desc_advance(identdesc, kk * 32), idesc, kk != 0);
#pragma unroll
              for (int kk = 0; kk < HDP / 16; ++kk)
                umma_bf16_ss(d, umma_desc_advance(adesc, kk * 32), umma_desc_advance(bdesc, kk * 32), idesc, 1);
              umma_commit(&sm.s_full[wg]);
            }
          }
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (leader && alive) umma_commit(&sm.q_empty[qb]);  // every product with these queries has been issued
      }
    }
  } else {
    if (NWG > 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::SOFTMAX_REGS));
    const int wg = (warp - 4) >> 2, quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t t_wg = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + wg * C::TM_WG;
    int stage = 0;
    uint32_t phase = 0, g = 0;
    bool alive = true;
    for (uint32_t item = blockIdx.x; item < p.total_items; item += gridDim.x) {
      float m_run = -INFINITY, l_run = 0.f;
      // (a step of COLS keys, as above)
      auto step = [&](auto width, int t) -> bool {
        constexpr int COLS = decltype(width)::value;
        const bool st_there = mbar_test(&sm.st_full[stage], phase), s_there = mbar_test(&sm.s_full[wg], g & 1);
        alive = (st_there || mbar_wait(&sm.st_full[stage], phase, p.status, ST_TIMEOUT_SOFTMAX)) &&
                (s_there || mbar_wait(&sm.s_full[wg], g & 1, p.status, ST_TIMEOUT_SOFTMAX));
        if (!__all_sync(0xffffffffu, alive)) {
          alive = false;
          return false;
        }
        tc_fence_after();
        const float mk0 = COLS >= 32 || lane < COLS ? sm.mb[stage][wg][lane] : 0.f;
        const float mk1 = COLS == 64 || lane + 32 < COLS ? sm.mb[stage][wg][lane + 32] : 0.f;
        float2 s[COLS / 2];
        {
          uint32_t r[COLS];
          if constexpr (COLS >= 32) tmem_ld32(t_wg, reinterpret_cast<uint32_t(&)[32]>(r));
          if constexpr (COLS == 64) tmem_ld32(t_wg + 32, reinterpret_cast<uint32_t(&)[32]>(r[32]));
          if constexpr (COLS % 32 == 16) tmem_ld16(t_wg + COLS - 16, reinterpret_cast<uint32_t(&)[16]>(r[COLS - 16]));
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < COLS / 2; ++e) s[e] = make_float2(__uint_as_float(r[2 * e]), __uint_as_float(r[2 * e + 1]));
        }
        if (__any_sync(0xffffffffu, mk0 != 0.f || mk1 != 0.f)) {
          const float* mrow = sm.mb[stage][wg];
#pragma unroll
          for (int c = 0; c < COLS / 4; ++c) {
            const float4 m4 = *reinterpret_cast<const float4*>(mrow + 4 * c);
            s[2 * c] = __fadd2_rn(s[2 * c], make_float2(m4.x, m4.y));
            s[2 * c + 1] = __fadd2_rn(s[2 * c + 1], make_float2(m4.z, m4.w));
            if ((c & 3) == 3) asm volatile("" ::: "memory");  // keep the loads from piling up in registers
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.st_empty[stage]);
        float mxa = fmaxf(s[0].x, s[0].y), mxb = fmaxf(s[1].x, s[1].y);
        float mxc = fmaxf(s[2].x, s[2].y), mxd = fmaxf(s[3].x, s[3].y);
#pragma unroll
        for (int e = 4; e < COLS / 2; e += 4) {
          mxa = fmax3(mxa, s[e].x, s[e].y);
          mxb = fmax3(mxb, s[e + 1].x, s[e + 1].y);
          mxc = fmax3(mxc, s[e + 2].x, s[e + 2].y);
          mxd = fmax3(mxd, s[e + 3].x, s[e + 3].y);
        }
        const float mx = fmaxf(fmaxf(mxa, mxb), fmaxf(mxc, mxd));
        const bool need = mx - m_run > RESCALE;  // true on the first step
        if (__any_sync(0xffffffffu, need)) {     // the offset moves only where the maximum grew a lot
          float scale = 1.0f;
          if (need) {
            const float off = rintf(m_run * LOG2E), off_new = rintf(mx * LOG2E);
            // (0 on the first step; beyond integers, offsets are the maxima themselves)
            scale = fast_exp2(fminf(fabsf(off), fabsf(off_new)) < INTEGER_OFFSETS ? off - off_new : (m_run - mx) * LOG2E);
            m_run = mx;
            l_run *= scale;
          }
          __syncwarp();
          if (t > 0) {
#pragma unroll
            for (int part = 0; part < HDP / 16; ++part) {
              uint32_t r[16];
              tmem_ld16(t_wg + C::TM_O + part * 16, r);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * scale);
              tmem_st16(t_wg + C::TM_O + part * 16, r);
            }
          }
        }
        // e^(s - m) = 2^(s log2e - offset): the product is exact in the fma and the offset an integer
        float minus_off = -rintf(m_run * LOG2E);
        if (__any_sync(0xffffffffu, fabsf(minus_off) >= INTEGER_OFFSETS)) {
          float2 minus_m = make_float2(0.f, 0.f);
          if (fabsf(minus_off) >= INTEGER_OFFSETS) {
            minus_m = make_float2(-m_run, -m_run);
            minus_off = 0.f;
          }
#pragma unroll
          for (int e = 0; e < COLS / 2; ++e) s[e] = __fadd2_rn(s[e], minus_m);
          __syncwarp();
        }
        const float2 log2e2 = make_float2(LOG2E, LOG2E), off2 = make_float2(minus_off, minus_off);
        float2 l2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int half = 0; half < COLS / 16; ++half) {
          uint32_t pc[3][8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float2 x = __ffma2_rn(s[half * 8 + e], log2e2, off2);
            const float2 w = make_float2(fast_exp2(x.x), fast_exp2(x.y));
            l2[e & 1] = __fadd2_rn(l2[e & 1], w);
            split3n2(w, pc[0][e], pc[1][e], pc[2][e]);
          }
#pragma unroll
          for (int q = 0; q < 3; ++q) tmem_st8(t_wg + C::TM_P + q * 32 + half * 8, pc[q]);
        }
        l_run += (l2[0].x + l2[0].y) + (l2[1].x + l2[1].y);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.p_full[wg]);
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
        return true;
      };
      const int whole = LAST < KT ? p.steps - 1 : p.steps;
      for (int t = 0; t < whole; ++t, ++g)
        if (!step(std::integral_constant<int, KT>{}, t)) break;
      if constexpr (LAST < KT) {
        if (alive) step(std::integral_constant<int, LAST>{}, whole);
        ++g;
      }
      alive = alive && mbar_wait(&sm.pv_done[wg], (g & 1) ^ 1, p.status, ST_TIMEOUT_SOFTMAX);
      if (!__all_sync(0xffffffffu, alive)) break;
      tc_fence_after();
      int b, h, i, j0;
      locate(item, b, h, i, j0);
      i += wg;
      const int j = j0 + row;
      const bool live = i < p.n_i && j < p.n;
      __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.o) +
                           ((static_cast<long long>(b * p.n_i + i) * p.n + j) * p.heads + h) * p.head_dim;
      const float inv = 1.0f / l_run;
#pragma unroll
      for (int part = 0; part < HDP / 16; ++part) {
        __syncwarp();
        uint32_t r[16];
        tmem_ld16(t_wg + C::TM_O + part * 16, r);
        tmem_ld_wait();
        if (!live) continue;
        uint4 w[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t u[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            u[e] = pack_bf16x2(__uint_as_float(r[8 * q + 2 * e]) * inv, __uint_as_float(r[8 * q + 2 * e + 1]) * inv);
          w[q] = make_uint4(u[0], u[1], u[2], u[3]);
        }
        uint4* dst = reinterpret_cast<uint4*>(out + part * 16);
        if (p.head_dim % 16 == 0 && part * 16 < p.head_dim) {
          store_sector(dst, w[0], w[1]);
        } else {
#pragma unroll
          for (int q = 0; q < 2; ++q)
            if (part * 16 + q * 8 < p.head_dim) dst[q] = w[q];
        }
      }
      __syncwarp();
      tc_fence_before();
    }
  }

  if (*reinterpret_cast<volatile int*>(p.status) != ST_OK)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

template <int HDP, int NWG>
int launch_bf16(const Maps& tm, Params p, bool pdl, cudaStream_t stream) {
  using C = BfCfg<HDP, NWG>;
  p.groups = (p.n_i + NWG - 1) / NWG;
  p.tiles_j = (p.n + 127) / 128;
  const long long items = static_cast<long long>(p.total_items) * p.groups * p.tiles_j;
  B200_REQUIRE(items < (1ll << 32) - 1024, B200TRI_ERR_UNSUPPORTED, "general attention: too many tiles");
  p.total_items = static_cast<uint32_t>(items);
  return with_last_columns<HDP <= 32 ? INT_MAX : 0>(p, [&](auto last) {
    const auto kernel = att_bf16_kernel<HDP, NWG, decltype(last)::value>;
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), (int)sizeof(BfSmem<HDP, NWG>));
    if (rc) return rc;
    const unsigned sms = sm_count(), grid = p.total_items < sms ? p.total_items : sms;
    return launch(kernel, dim3(grid), dim3(C::THREADS), sizeof(BfSmem<HDP, NWG>), stream, pdl, tm, p);
  });
}

// Rows of an item. A step of four takes some 1.2 times as long as one of three, which pays
// unless as many rounds of items are needed: 12 heads x 100 tokens, attention 58.8 us with four and 55.7 with three
// (three rounds either way), 4 x 4 heads x 200 tokens 173 and 183 (11 and 15 rounds). (Over 91 shapes of 20 to 320
// tokens the rule takes the faster or loses up to 5 %, most with one or two rounds of one step.)
template <int HDP>
int launch_bf16_narrow(const Maps& tm, const Params& p, bool pdl, cudaStream_t stream) {
  auto rounds = [&](int rows) {
    const long long items = static_cast<long long>(p.total_items) * ((p.n_i + rows - 1) / rows) * ((p.n + 127) / 128);
    return (items + sm_count() - 1) / sm_count();
  };
  return 5 * rounds(3) < 6 * rounds(4) ? launch_bf16<HDP, 3>(tm, p, pdl, stream) : launch_bf16<HDP, 4>(tm, p, pdl, stream);
}

}  // namespace

int launch_att_split(const AttSplitArgs& a, cudaStream_t stream) {
  B200_REQUIRE(a.head_dim % 8 == 0 && a.head_dim >= 8 && a.head_dim <= 64, B200TRI_ERR_UNSUPPORTED,
               "general attention: head widths are multiples of 8 up to 64 (got %d)", a.head_dim);
  const bool token = a.pieces != nullptr;
  B200_REQUIRE(!token || (!a.bf16 && a.batch == 1 && a.n_i == 1 && a.head_dim <= 32), B200TRI_ERR_INVALID,
               "general attention: the gated form takes one row of heads up to 32 wide");
  const uint32_t hdp = a.bf16 && a.head_dim <= 16 ? 16 : a.head_dim <= 32 ? 32 : 64;
  const Swz qk_swz = hdp == 16 ? Swz::B32 : hdp == 32 ? Swz::B64 : Swz::B128;
  const uint64_t hd = a.head_dim, heads = a.heads, width = hd * heads, n = a.n;
  const uint64_t rows = static_cast<uint64_t>(a.n_i) * a.batch, in = a.bf16 ? 1 : 3;
  Maps tm;
  int rc;
  {
    const uint64_t dims[5] = {hd, heads, n, rows, in};
    const uint64_t str[4] = {hd * 2, width * 2, n * width * 2, rows * n * width * 2};
    const uint32_t box_q[5] = {hdp, 1, 128, 1, 1}, box_k[5] = {hdp, 1, KT, 1, 1};
    if ((rc = make_tmap(&tm.q, a.q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box_q, qk_swz))) return rc;
    if ((rc = make_tmap(&tm.k, a.k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box_k, qk_swz))) return rc;
  }
  {
    const uint64_t ld = a.v_ld;
    const uint64_t dims[5] = {n, hd, heads, rows, in};
    const uint64_t str[4] = {ld * 2, hd * ld * 2, width * ld * 2, rows * width * ld * 2};
    const uint32_t box[5] = {KT, hdp, 1, 1, 1};
    if ((rc = make_tmap(&tm.v, a.vt, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box, Swz::B128))) return rc;
  }
  {
    const uint64_t ld = a.bias_ld, size = a.bf16 ? 2 : 4;
    const uint64_t dims[4] = {n, n, heads, static_cast<uint64_t>(a.batch)};
    const uint64_t str[3] = {ld * size, n * ld * size, heads * n * ld * size};
    const uint32_t box[4] = {a.bf16 ? 64u : 32u, 128, 1, 1};
    if ((rc = make_tmap(&tm.b, a.bias, a.bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dims, str,
                        box, Swz::B128)))
      return rc;
  }
  {
    const uint64_t ld = a.mask_ld;
    const uint64_t dims[2] = {ld, rows};
    const uint64_t str[1] = {ld * 4};
    const uint32_t box[2] = {KT, 1};
    if ((rc = make_tmap(&tm.m, a.mask_bias, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, dims, str, box, Swz::None))) return rc;
  }
  Params p = {};
  p.n_i = a.n_i;
  p.n = a.n;
  p.heads = a.heads;
  p.head_dim = a.head_dim;
  p.steps = (a.n + KT - 1) / KT;
  p.total_items = static_cast<uint32_t>(a.batch) * a.heads;
  p.scale = a.scale;
  p.o = a.o;
  p.gate = a.gate;
  p.pieces = a.pieces;
  p.status = device_status_word();
  B200_REQUIRE(p.status != nullptr, B200TRI_ERR_CUDA, "general attention: no current CUDA device");
  // One row: tiles of 128 queries in a CTA of their own where the SMs are enough for all. A step is 36 products of the tensor pipe
  // a tile, and with two tiles to a CTA they queued for each other: 203 / 1024 tokens 18.9 / 56.2 us, 13.9 / 40.5 so (blocks of 128 /
  // 203 / 300 tokens 157.1 / 260.3 / 473.2 -> 155.0 / 255.6 / 465.6). With more tiles than SMs two share their keys.
  if (token)
    return static_cast<long long>(a.heads) * ((a.n + 127) / 128) <= sm_count() ? launch_cfg<32, true, 1>(tm, p, a.pdl, stream)
                                                                               : launch_cfg<32, true, 2>(tm, p, a.pdl, stream);
  if (a.bf16 && hdp == 16) return launch_bf16_narrow<16>(tm, p, a.pdl, stream);
  if (a.bf16) return hdp == 32 ? launch_bf16_narrow<32>(tm, p, a.pdl, stream) : launch_bf16<64, 2>(tm, p, a.pdl, stream);
  return hdp == 32 ? launch_cfg<32, false, 2>(tm, p, a.pdl, stream) : launch_cfg<64, false, 1>(tm, p, a.pdl, stream);
}

}  // namespace b200
