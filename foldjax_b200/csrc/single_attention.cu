// Single-representation attention with pair bias (the block's other consumer of z).
//
//   q = s @ Wq + bq,  g = sigmoid(s @ Wg),  k = k_in @ Wk,  v = k_in @ Wv
//   bias[h,i,j] = LN(z[i,j,:]) @ Wz[:,h]                      (z read once, in fp32)
//   out = (g * softmax_j(q_h . k_h / sqrt(d) + bias + (1 - mask_j) * -inf) v_h) @ Wo
//
// Reference: attention_pair_bias_forward,
// src/foldjax/models/boltz2/models/primitives/attention.py:19-140 (XLA branch
// :85-110, _attention_qblock :124-140), called from the Pairformer block with
// s and z in float32, src/foldjax/models/boltz2/models/trunk_blocks/pairformer.py:188-203.
// Everything here is fp32 arithmetic on fp32 s and bf16 z / weights (the trunk
// dtype), like the reference's promoted computation.
//
// The pass over z is pair_bias_kernel, bound by HBM (256 B read and 4 * heads B written per pair);
// the token attention is att_split.cu's one-row form; the products are gemm.cuh's.
#include "att_split.cuh"
#include "host.cuh"
#include "single.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int C_Z = 128;
constexpr int MAX_HEADS = 16;
constexpr int HD = 24;  // head width the token-attention kernel is built for

// ---------------------------------------------------------------- pair bias
// Tiles of 128 pairs. With gamma folded into the projection,
//   bias_h = rstd * (sum_c x_c W'[c][h] - mean * sum_c W'[c][h]) + sum_c beta_c W[c][h],
// so the normalised row is never formed. x is bf16 already and W' goes in as three bf16 pieces, 16
// columns each, so one 128 x 48 x 128 product on the tensor cores is as exact as a float32 one;
// meanwhile one thread per pair takes mean and variance (two-pass, as the reference computes
// them) from the same shared-memory tile. On the CUDA cores the 2048 multiply-adds of a pair
// were the bound: 200 us at n = 1024, four times what the bytes need.
//   warps 0-3   mean, variance, result     warp 4   TMA producer     warp 5   MMA issuer
// Two CTAs per SM: one's loads and result stores run beside the other's arithmetic.
constexpr int PB_STAGES = 3, PB_TILE = 128 * C_Z * 2, PB_N = 3 * MAX_HEADS, PB_W = PB_N * 128;
constexpr int PB_THREADS = 192, PB_SMEM = PB_STAGES * PB_TILE + 2 * PB_W + 1024;

struct PairBiasParams {
  uint32_t n_pairs, n;
  int ld, heads, mask_ld;
  bool early;  // the weights may be read before the predecessor in the stream is through
  const __nv_bfloat16 *ln_scale, *ln_bias, *wz;
  float eps, inf;
  const float* mask;
  float *bias, *mask_rows;
  int* status;
};

__global__ void __launch_bounds__(PB_THREADS, 2) pair_bias_kernel(const __grid_constant__ CUtensorMap tm_z, const PairBiasParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* w_s = smem + PB_STAGES * PB_TILE;  // W' pieces, K-major: two halves of 64 channels x 48 rows
  __shared__ uint64_t full_bar[PB_STAGES], empty_bar[PB_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ float sw[MAX_HEADS], bw[MAX_HEADS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tm_z);
    for (int s = 0; s < PB_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1 + 4);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    fence_barrier_init();
  }
  if (warp == 5) {
    tmem_alloc(&tmem_base_s, 128);
    tmem_relinquish();
  }
  if (!p.early) pdl_wait();
  if (warp < 4) {  // thread = (head, 16 channels)
    const int h = threadIdx.x >> 3, c0 = (threadIdx.x & 7) * 16;
    float sum = 0.f, beta = 0.f;
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      float w[2] = {0.f, 0.f};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = c0 + e + u;
        const float raw = h < p.heads ? __bfloat162float(p.wz[c * p.heads + h]) : 0.f;
        w[u] = __bfloat162float(p.ln_scale[c]) * raw;
        sum += w[u];
        beta += __bfloat162float(p.ln_bias[c]) * raw;
      }
      uint32_t pc[3];
      split3x2(w[0], w[1], pc[0], pc[1], pc[2]);
      const int k = (c0 + e) & 63;
#pragma unroll
      for (int q = 0; q < 3; ++q)
        *reinterpret_cast<uint32_t*>(w_s + (c0 >> 6) * PB_W + sw128_offset(q * MAX_HEADS + h, k >> 3) + (k & 7) * 2) = pc[q];
    }
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
      sum += __shfl_xor_sync(0xffffffffu, sum, d);
      beta += __shfl_xor_sync(0xffffffffu, beta, d);
    }
    if ((threadIdx.x & 7) == 0) {
      sw[h] = sum;
      bw[h] = beta;
    }
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (p.early) pdl_wait();
  pdl_trigger();
  const uint32_t tmem_base = tmem_base_s;
  const uint32_t tiles = (p.n_pairs + 127) / 128;

  if (warp == 4) {
    if (elect_one()) {
      uint32_t it = 0;
      for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
        const uint32_t stage = it % PB_STAGES;
        if (!mbar_wait(&empty_bar[stage], ((it / PB_STAGES) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
        uint8_t* dst = smem + stage * PB_TILE;
        mbar_expect_tx(&full_bar[stage], PB_TILE);
        for (int half = 0; half < 2; ++half)
          tma_load_2d(dst + half * (PB_TILE / 2), &tm_z, &full_bar[stage], half * 64, static_cast<int>(tile * 128));
      }
    }
  } else if (warp == 5) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, PB_N);
      uint32_t it = 0;
      for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
        const uint32_t stage = it % PB_STAGES, buf = it & 1;
        if (!mbar_wait(&acc_empty[buf], ((it >> 1) & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) break;
        if (!mbar_wait(&full_bar[stage], (it / PB_STAGES) & 1, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint64_t adesc = umma_desc_kmajor(smem_u32(smem + stage * PB_TILE + half * (PB_TILE / 2)), 128);
          const uint64_t bdesc = umma_desc_kmajor(smem_u32(w_s + half * PB_W), 128);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ss(tmem_base + buf * 64, umma_desc_advance(adesc, k * 32), umma_desc_advance(bdesc, k * 32), idesc,
                         (half | k) != 0);
        }
        umma_commit(&empty_bar[stage]);
        umma_commit(&acc_full[buf]);
      }
    }
  } else {
    // the token attention's mask row; keys past the end get no weight
    if (blockIdx.x == 0)
      for (int j = threadIdx.x; j < p.mask_ld; j += 128)
        p.mask_rows[j] = j < static_cast<int>(p.n) ? fmaxf((1.0f - p.mask[j]) * -p.inf, SPLIT_MASK_MIN) : SPLIT_MASK_PAD;
    const int r = threadIdx.x;
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
      const uint32_t stage = it % PB_STAGES, buf = it & 1;
      if (!mbar_wait(&full_bar[stage], (it / PB_STAGES) & 1, p.status, ST_TIMEOUT_EPILOGUE)) break;
      const uint8_t* src = smem + stage * PB_TILE;
      uint4 x[16];
      float2 s4[4] = {};
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        x[c] = *reinterpret_cast<const uint4*>(src + (c >> 3) * (PB_TILE / 2) + sw128_offset(r, c & 7));
        s4[0] = __fadd2_rn(s4[0], make_float2(bf16_lo(x[c].x), bf16_hi(x[c].x)));
        s4[1] = __fadd2_rn(s4[1], make_float2(bf16_lo(x[c].y), bf16_hi(x[c].y)));
        s4[2] = __fadd2_rn(s4[2], make_float2(bf16_lo(x[c].z), bf16_hi(x[c].z)));
        s4[3] = __fadd2_rn(s4[3], make_float2(bf16_lo(x[c].w), bf16_hi(x[c].w)));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[stage]);
      const float2 s2 = __fadd2_rn(__fadd2_rn(s4[0], s4[1]), __fadd2_rn(s4[2], s4[3]));
      const float mean = (s2.x + s2.y) * (1.0f / C_Z);
      const float2 mm = make_float2(-mean, -mean);
      float2 q4[4] = {};
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const uint32_t v[4] = {x[c].x, x[c].y, x[c].z, x[c].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 d = __fadd2_rn(make_float2(bf16_lo(v[e]), bf16_hi(v[e])), mm);
          q4[e] = __ffma2_rn(d, d, q4[e]);
        }
      }
      const float2 q2 = __fadd2_rn(__fadd2_rn(q4[0], q4[1]), __fadd2_rn(q4[2], q4[3]));
      const float rstd = rsqrtf((q2.x + q2.y) * (1.0f / C_Z) + p.eps);
      if (!mbar_wait(&acc_full[buf], (it >> 1) & 1, p.status, ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      __syncwarp();
      uint32_t hi[16], mid[16], lo[16];
      const uint32_t t = tmem_base + (static_cast<uint32_t>(warp * 32) << 16) + buf * 64;
      tmem_ld16(t, hi);
      tmem_ld16(t + 16, mid);
      tmem_ld16(t + 32, lo);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
      const uint32_t pair = tile * 128 + r;
      if (pair < p.n_pairs) {
        const uint32_t i = pair / p.n, j = pair - i * p.n;
        float* dst = p.bias + static_cast<size_t>(i) * p.ld + j;
        const size_t plane = static_cast<size_t>(p.n) * p.ld;
#pragma unroll
        for (int h = 0; h < MAX_HEADS; ++h)
          if (h < p.heads) {
            const float dot = __uint_as_float(hi[h]) + (__uint_as_float(mid[h]) + __uint_as_float(lo[h]));
            dst[h * plane] = rstd * (dot - mean * sw[h]) + bw[h];
          }
      }
    }
  }

  if (*reinterpret_cast<volatile int*>(p.status) != ST_OK)
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem_base, 128);
}

// ------------------------------------------------------------------ row kernels
// See launch_row_norm. One block per row, four neighbouring channels per thread: every load of a
// row (the base and up to eight partial planes) is in flight at once. With one warp per row and
// the planes added one after the other the kernel was a chain of 96 dependent loads, 20 us.
constexpr int ROW_THREADS = MAX_HEADS * HD / 4;
__device__ __forceinline__ float row_sum(float v, float* scratch) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  return (scratch[0] + scratch[1]) + scratch[2];
}
// `aligned`: base and sum_out, the caller's tensors, start on a 16-byte boundary (rows are 32 bytes
// apart or a multiple of that; the partials lie in the workspace).
__global__ void __launch_bounds__(ROW_THREADS) row_norm_kernel(const RowArgs a, const bool aligned) {
  static_assert(ROW_THREADS == 96, "three warps");
  __shared__ float scratch[2][3];
  pdl_wait();
  pdl_trigger();
  const int row = blockIdx.x, i = threadIdx.x * 4;
  const bool live = i < a.c;  // c is a multiple of 8
  const long long off = static_cast<long long>(row) * a.c + i, plane = static_cast<long long>(a.rows) * a.c;
  const bool keep = a.row_mask == nullptr || a.row_mask[row] != 0.f;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (live && keep) {
    float4 part[SINGLE_MAX_SPLITS], base = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int p = 0; p < SINGLE_MAX_SPLITS; ++p)
      part[p] = a.partial && p < a.splits ? *reinterpret_cast<const float4*>(a.partial + p * plane + off)
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.base) {
      const float* src = a.base + off;
      base = aligned ? *reinterpret_cast<const float4*>(src) : make_float4(src[0], src[1], src[2], src[3]);
    }
#pragma unroll
    for (int p = 0; p < SINGLE_MAX_SPLITS; ++p) {
      v[0] += part[p].x;
      v[1] += part[p].y;
      v[2] += part[p].z;
      v[3] += part[p].w;
    }
    v[0] = base.x + v[0];
    v[1] = base.y + v[1];
    v[2] = base.z + v[2];
    v[3] = base.w + v[3];
  }
  if (a.sum_out && live) {
    if (aligned) {
      *reinterpret_cast<float4*>(a.sum_out + off) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) a.sum_out[off + e] = v[e];
    }
  }
  if (!a.pieces) return;
  if (a.scale) {
    const float mean = row_sum((v[0] + v[1]) + (v[2] + v[3]), scratch[0]) / a.c;
    float q = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) q += live ? (v[e] - mean) * (v[e] - mean) : 0.f;
    const float rstd = 1.0f / sqrtf(row_sum(q, scratch[1]) / a.c + a.eps);
    const __nv_bfloat16* scale = static_cast<const __nv_bfloat16*>(a.scale);
    const __nv_bfloat16* bias = static_cast<const __nv_bfloat16*>(a.bias);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (live) v[e] = (v[e] - mean) * rstd * __bfloat162float(scale[i + e]) + __bfloat162float(bias[i + e]);
  }
  if (!live) return;
  uint32_t pc[3][2];
  split3x2(v[0], v[1], pc[0][0], pc[1][0], pc[2][0]);
  split3x2(v[2], v[3], pc[0][1], pc[1][1], pc[2][1]);
#pragma unroll
  for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(a.pieces + q * plane + off) = make_uint2(pc[q][0], pc[q][1]);
}

// dst[k][ld] = src[k][n], padding columns zero: weights TMA cannot read as they are.
__global__ void pad_weight_kernel(const __nv_bfloat16* __restrict__ src, int k, int n, int ld,
                                  __nv_bfloat16* __restrict__ dst) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= static_cast<long long>(k) * ld) return;
  const int r = static_cast<int>(idx / ld), c = static_cast<int>(idx % ld);
  dst[idx] = c < n ? src[static_cast<long long>(r) * n + c] : __float2bfloat16_rn(0.f);
}

// ---------------------------------------------------------------- product policies
// float32 activations (three pieces) x bf16 weights as stored. The products of a block are
// 0.6-15 GFLOP, so what bounds them at every size is latency: many small tiles, K split until the
// tiles cover the SMs. (128 x 384 x 384 in 64 x 64 tiles without a split - six blocks on the whole
// chip, 24 dependent k steps - is 116 us on the CUDA cores.)
//
// [q | k | v | g] in one launch: column tiles of 64 walk the four weights in turn. q and k leave as
// pieces, v as transposed pieces (both as the token attention reads them), the gate in float32.
struct QkvgPolicy : NoPrefetch {
  static constexpr int BN = 64, PA = 3, PB = 1, NSEG = 1, NMAIN = 3;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = 8, CTAS = 1;
  struct Params {
    int rows, c, tiles_per_w, first_w;
    long long v_ld;
    const __nv_bfloat16* q_bias;
    __nv_bfloat16 *q, *k, *vt;
    float* gate;
  };
  static __device__ void load_a(const GemmMaps& maps, const Params&, int, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    tma_load_3d(dst, &maps.a[0], bar, k, m_tile * GEMM_BM, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params& p, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    gemm_load_mn(&maps.b[p.first_w + n_tile / p.tiles_per_w], dst, bar, 1, n_tile % p.tiles_per_w * BN, k, piece);
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<QkvgPolicy>& acc, int quarter,
                                  int col0, int col1, int lane, const Pre&) {
    const int row = m_tile * GEMM_BM + quarter * 32 + lane;
    const int which = p.first_w + n_tile / p.tiles_per_w;
    const long long plane = static_cast<long long>(p.rows) * p.c, off = static_cast<long long>(row) * p.c;
#pragma unroll 1
    for (int col = col0; col < col1; col += 16) {
      float r[16];
      acc.load(0, col, r);
      const int c0 = n_tile % p.tiles_per_w * BN + col;
      if (row >= p.rows || c0 >= p.c) continue;
      if (which == 2) {  // one channel per store: 32 lanes are 32 neighbouring tokens
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (c0 + e >= p.c) break;  // c is a multiple of 8
          __nv_bfloat16* dst = p.vt + (c0 + e) * p.v_ld + row;
          split3(r[e], dst[0], dst[p.c * p.v_ld], dst[2 * p.c * p.v_ld]);
        }
        continue;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int c8 = c0 + 8 * q;
        if (c8 >= p.c) break;
        float* v = r + 8 * q;
        if (which == 3) {
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = 1.0f / (1.0f + expf(-v[e]));
          float4* dst = reinterpret_cast<float4*>(p.gate + off + c8);
          dst[0] = make_float4(v[0], v[1], v[2], v[3]);
          dst[1] = make_float4(v[4], v[5], v[6], v[7]);
          continue;
        }
        uint32_t pc[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (which == 0) {
            v[2 * e] += __bfloat162float(p.q_bias[c8 + 2 * e]);
            v[2 * e + 1] += __bfloat162float(p.q_bias[c8 + 2 * e + 1]);
          }
          split3x2(v[2 * e], v[2 * e + 1], pc[0][e], pc[1][e], pc[2][e]);
        }
        __nv_bfloat16* dst = (which == 0 ? p.q : p.k) + off + c8;
#pragma unroll
        for (int t = 0; t < 3; ++t)
          *reinterpret_cast<uint4*>(dst + t * plane) = make_uint4(pc[t][0], pc[t][1], pc[t][2], pc[t][3]);
      }
    }
  }
};

// float32 partial sums, one plane per K split.
struct PartialPolicy : NoPrefetch {
  static constexpr int BN = 64, PA = 3, PB = 1, NSEG = 1, NMAIN = 3;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = 8, CTAS = 1;
  struct Params {
    int rows, n;
    float* out;
  };
  static __device__ void load_a(const GemmMaps& maps, const Params&, int, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    tma_load_3d(dst, &maps.a[0], bar, k, m_tile * GEMM_BM, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params&, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    gemm_load_mn(&maps.b[0], dst, bar, 1, n_tile * BN, k, piece);
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int split, const Accum<PartialPolicy>& acc,
                                  int quarter, int col0, int col1, int lane, const Pre&) {
    const int row = m_tile * GEMM_BM + quarter * 32 + lane;
#pragma unroll 1
    for (int col = col0; col < col1; col += 16) {
      float r[16];
      acc.load(0, col, r);
      if (row >= p.rows) continue;
      const int c0 = n_tile * BN + col;
      float* dst = p.out + (static_cast<long long>(split) * p.rows + row) * p.n + c0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (c0 + 4 * q < p.n)
          *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
    }
  }
};

// 64 columns of x @ fc1 beside the same 64 of x @ fc2; silu(a) * b leaves as pieces
// (transition.py:108).
struct SwigluPolicy : NoPrefetch {
  static constexpr int BN = 128, PA = 3, PB = 1, NSEG = 1, NMAIN = 3;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = 8, CTAS = 1;
  struct Params {
    int rows, hidden;
    long long pitch;  // of a piece's rows
    __nv_bfloat16* h;
  };
  static __device__ void load_a(const GemmMaps& maps, const Params&, int, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    tma_load_3d(dst, &maps.a[0], bar, k, m_tile * GEMM_BM, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params&, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    for (int w = 0; w < 2; ++w) gemm_load_mn(&maps.b[w], dst + w * 8192, bar, 1, n_tile * 64, k, piece);
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<SwigluPolicy>& acc, int quarter,
                                  int col0, int col1, int lane, const Pre&) {
    const int row = m_tile * GEMM_BM + quarter * 32 + lane;
    const long long plane = static_cast<long long>(p.rows) * p.pitch;
#pragma unroll 1
    for (int col = col0 / 2; col < col1 / 2; col += 16) {  // this warp's share of the 64 hidden columns
      float a[16], b[16];
      acc.load(0, col, a);
      acc.load(0, 64 + col, b);
      if (row >= p.rows) continue;
      const int c0 = n_tile * 64 + col;
      __nv_bfloat16* dst = p.h + static_cast<long long>(row) * p.pitch + c0;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (c0 + 8 * q >= p.pitch) break;  // the pitch is a multiple of 8; padding columns come out as zero
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float v[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float av = a[8 * q + 2 * e + u];
            v[u] = av / (1.0f + expf(-av)) * b[8 * q + 2 * e + u];
          }
          split3x2(v[0], v[1], hi[e], mid[e], lo[e]);
        }
        *reinterpret_cast<uint4*>(dst + 8 * q) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(dst + plane + 8 * q) = make_uint4(mid[0], mid[1], mid[2], mid[3]);
        *reinterpret_cast<uint4*>(dst + 2 * plane + 8 * q) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      }
    }
  }
};

}  // namespace

int launch_row_norm(const RowArgs& a, cudaStream_t stream, bool pdl) {
  const bool aligned = ((reinterpret_cast<uintptr_t>(a.base) | reinterpret_cast<uintptr_t>(a.sum_out)) & 15) == 0;
  return launch(row_norm_kernel, dim3(a.rows), dim3(ROW_THREADS), 0, stream, pdl, a, aligned);
}

// Enough splits that the tiles cover the SMs, at least two k steps each, none of them empty. A B200's
// SM count and not the limit that may be set on it: the splits are float32 sums of their own, and the
// bits of a result are not to depend on how many SMs it was computed on.
int single_splits(int tiles, int kb) {
  constexpr int SMS = 148;
  int s = SMS / (tiles > 0 ? tiles : 1);
  s = s > kb / 2 ? kb / 2 : s;
  s = s > SINGLE_MAX_SPLITS ? SINGLE_MAX_SPLITS : s;
  if (s <= 1) return 1;
  const int per = (kb + s - 1) / s;
  return (kb + per - 1) / per;
}

size_t tma_weight_bytes(int k, int n) { return static_cast<size_t>(k) * round_up(n, 8) * 2; }

int tma_weight(const void* w, int k, int n, void* scratch, cudaStream_t stream, const void** out, long long* pitch) {
  *out = w;
  *pitch = n;
  if (n % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) return B200TRI_OK;
  *out = scratch;
  *pitch = round_up(n, 8);
  const long long total = static_cast<long long>(k) * *pitch;
  return launch(pad_weight_kernel, dim3(static_cast<unsigned>((total + 255) / 256)), dim3(256), 0, stream, false,
                static_cast<const __nv_bfloat16*>(w), k, n, static_cast<int>(*pitch), static_cast<__nv_bfloat16*>(scratch));
}

static int kblocks(int k) { return (k + GEMM_BK - 1) / GEMM_BK; }
static int mtiles(int rows) { return (rows + GEMM_BM - 1) / GEMM_BM; }

int launch_linear_partial(const __nv_bfloat16* pieces, long long pitch, int rows, int k, const void* w, int n,
                          void* w_scratch, float* partial, int* splits, cudaStream_t stream, bool pdl) {
  const void* wp;
  long long wpitch;
  int rc = tma_weight(w, k, n, w_scratch, stream, &wp, &wpitch);
  if (rc) return rc;
  GemmMaps maps = {};
  if ((rc = gemm_map_kmajor(&maps.a[0], pieces, 3, rows, k, pitch, GEMM_BM))) return rc;
  if ((rc = gemm_map_mnmajor(&maps.b[0], wp, k, n, wpitch))) return rc;
  GemmShape g = {mtiles(rows), (n + PartialPolicy::BN - 1) / PartialPolicy::BN, 1, {kblocks(k), 0}, nullptr};
  g.splits = single_splits(g.m_tiles * g.n_tiles, g.kb[0]);
  *splits = g.splits;
  return launch_piece_gemm<PartialPolicy>(maps, g, {rows, n, partial}, stream, pdl && wp == w);
}

int launch_swiglu(const __nv_bfloat16* pieces, int rows, int k, const void* fc1, const void* fc2, int hidden,
                  void* w1_scratch, void* w2_scratch, __nv_bfloat16* h, long long pitch, cudaStream_t stream, bool pdl) {
  const void *w1, *w2;
  long long p1, p2;
  int rc = tma_weight(fc1, k, hidden, w1_scratch, stream, &w1, &p1);
  if (rc || (rc = tma_weight(fc2, k, hidden, w2_scratch, stream, &w2, &p2))) return rc;
  GemmMaps maps = {};
  if ((rc = gemm_map_kmajor(&maps.a[0], pieces, 3, rows, k, k, GEMM_BM))) return rc;
  if ((rc = gemm_map_mnmajor(&maps.b[0], w1, k, hidden, p1))) return rc;
  if ((rc = gemm_map_mnmajor(&maps.b[1], w2, k, hidden, p2))) return rc;
  const GemmShape g = {mtiles(rows), (hidden + 63) / 64, 1, {kblocks(k), 0}, nullptr};
  return launch_piece_gemm<SwigluPolicy>(maps, g, {rows, hidden, pitch, h}, stream, pdl && w1 == fc1 && w2 == fc2);
}

SingleAttentionWork single_attention_work(int n, int c_s, int heads) {
  SingleAttentionWork w;
  Carver c(nullptr);
  const size_t act = static_cast<size_t>(n) * c_s;
  auto take = [&](size_t bytes) {
    c.take<uint8_t>(bytes);
    return c.off - bytes;
  };
  w.q = take(act * 2 * 3);
  w.k = take(act * 2 * 3);
  w.vt = take(static_cast<size_t>(c_s) * round_up(n, 8) * 2 * 3);
  w.g = take(act * 4);
  w.bias = take(static_cast<size_t>(heads) * n * round_up(n, 8) * 4);
  w.mask = take(static_cast<size_t>(round_up(n, 64)) * 4);
  w.ao = take(act * 2 * 3);
  for (size_t& off : w.w) off = take(tma_weight_bytes(c_s, c_s));
  w.total = c.total();
  return w;
}

namespace {
const __nv_bfloat16* bf(const void* p) { return static_cast<const __nv_bfloat16*>(p); }
}  // namespace

int single_project(const b200tri_attention_pair_bias_args* a, const __nv_bfloat16* xq, const __nv_bfloat16* xk, uint8_t* work,
                   cudaStream_t stream) {
  const int n = a->n, c_s = a->c_s;
  const SingleAttentionWork off = single_attention_work(n, c_s, a->heads);
  // With separate key-side rows: k, v from those in a launch of their own.
  const bool same = xq == xk;
  const void* w[4] = {a->proj_q, a->proj_k, a->proj_v, a->proj_g};
  GemmMaps maps = {};
  bool direct = true;
  int rc;
  for (int i = 0; i < 4; ++i) {
    const void* wp;
    long long pitch;
    if ((rc = tma_weight(w[i], c_s, c_s, work + off.w[i], stream, &wp, &pitch))) return rc;
    if ((rc = gemm_map_mnmajor(&maps.b[i], wp, c_s, c_s, pitch))) return rc;
    direct = direct && wp == w[i];
  }
  const int per_w = (c_s + QkvgPolicy::BN - 1) / QkvgPolicy::BN;
  auto at = [&](size_t o) { return reinterpret_cast<__nv_bfloat16*>(work + o); };
  QkvgPolicy::Params ep = {n,         c_s,       per_w,      0, round_up(n, 8), bf(a->proj_q_bias), at(off.q), at(off.k),
                           at(off.vt), reinterpret_cast<float*>(work + off.g)};
  // (first weight, weight count) of each launch
  const int runs_same[1][2] = {{0, 4}}, runs_split[3][2] = {{0, 1}, {1, 2}, {3, 1}};
  const int n_runs = same ? 1 : 3;
  for (int r = 0; r < n_runs; ++r) {
    const int* run = same ? runs_same[r] : runs_split[r];
    if ((rc = gemm_map_kmajor(&maps.a[0], !same && r == 1 ? xk : xq, 3, n, c_s, c_s, GEMM_BM))) return rc;
    ep.first_w = run[0];
    const GemmShape g = {mtiles(n), per_w * run[1], 1, {kblocks(c_s), 0}, nullptr};
    if ((rc = launch_piece_gemm<QkvgPolicy>(maps, g, ep, stream, direct && same))) return rc;
  }
  return B200TRI_OK;
}

int single_pair_bias(const b200tri_attention_pair_bias_args* a, uint8_t* work, cudaStream_t stream, bool pdl) {
  const int n = a->n;
  const SingleAttentionWork off = single_attention_work(n, a->c_s, a->heads);
  const long long n_pairs = static_cast<long long>(n) * n;
  B200_REQUIRE(n_pairs < (1ll << 31) - 128, B200TRI_ERR_UNSUPPORTED, "pair bias: too many tokens (%d)", n);
  PairBiasParams p = {};
  p.n_pairs = static_cast<uint32_t>(n_pairs);
  p.n = n;
  p.ld = round_up(n, 8);
  p.heads = a->heads;
  p.mask_ld = round_up(n, 64);
  p.early = pdl_chained();
  p.ln_scale = bf(a->proj_z_norm_scale);
  p.ln_bias = bf(a->proj_z_norm_bias);
  p.wz = bf(a->proj_z);
  p.eps = a->eps;
  p.inf = a->inf;
  p.mask = static_cast<const float*>(a->mask);
  p.bias = reinterpret_cast<float*>(work + off.bias);
  p.mask_rows = reinterpret_cast<float*>(work + off.mask);
  p.status = device_status_word();
  B200_REQUIRE(p.status != nullptr, B200TRI_ERR_CUDA, "pair bias: no current CUDA device");
  CUtensorMap tm_z;
  const uint64_t dims[2] = {C_Z, static_cast<uint64_t>(n_pairs)};
  const uint64_t str[1] = {C_Z * 2};
  const uint32_t box[2] = {64, 128};
  int rc = make_tmap(&tm_z, a->z, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dims, str, box, Swz::B128);
  if (rc || (rc = ensure_smem_limit(reinterpret_cast<const void*>(pair_bias_kernel), PB_SMEM))) return rc;
  const long long tiles = (n_pairs + 127) / 128, slots = 2ll * sm_count();
  TimedLaunch timed(K_PAIR_BIAS, stream);
  return launch(pair_bias_kernel, dim3(static_cast<unsigned>(tiles < slots ? tiles : slots)), dim3(PB_THREADS), PB_SMEM, stream,
                pdl, tm_z, p);
}

int single_attend(const b200tri_attention_pair_bias_args* a, uint8_t* work, float* partial, int* splits, cudaStream_t stream,
                  bool pdl) {
  const int n = a->n, c_s = a->c_s;
  const SingleAttentionWork off = single_attention_work(n, c_s, a->heads);
  AttSplitArgs s = {};
  s.batch = s.n_i = 1;
  s.n = n;
  s.heads = a->heads;
  s.head_dim = HD;
  s.q = bf(work + off.q);
  s.k = bf(work + off.k);
  s.vt = bf(work + off.vt);
  s.v_ld = s.bias_ld = round_up(n, 8);
  s.bias = work + off.bias;
  s.mask_bias = reinterpret_cast<float*>(work + off.mask);
  s.mask_ld = round_up(n, 64);
  s.scale = 1.0f / sqrtf(static_cast<float>(HD));
  s.gate = reinterpret_cast<float*>(work + off.g);
  s.pieces = reinterpret_cast<__nv_bfloat16*>(work + off.ao);
  s.pdl = pdl;
  const int rc = launch_att_split(s, stream);
  if (rc) return rc;
  return launch_linear_partial(s.pieces, c_s, n, c_s, a->proj_o, c_s, work + off.w[4], partial, splits, stream, true);
}

}  // namespace b200

// Standalone entry: the pieces of s (and of k_in), the attention, the sum of its partials.
namespace {
struct StandalonePlan {
  size_t xq, xk, partial, work, total;
};
StandalonePlan standalone_plan(int n, int c_s, int heads) {
  using namespace b200;
  StandalonePlan p;
  Carver c(nullptr);
  const size_t act = static_cast<size_t>(n) * c_s;
  auto take = [&](size_t bytes) {
    c.take<uint8_t>(bytes);
    return c.off - bytes;
  };
  p.xq = take(act * 2 * 3);
  p.xk = take(act * 2 * 3);
  p.partial = take(act * 4 * SINGLE_MAX_SPLITS);
  p.work = take(single_attention_work(n, c_s, heads).total);
  p.total = c.total();
  return p;
}
}  // namespace

extern "C" size_t b200tri_attention_pair_bias_workspace_bytes(int32_t n, int32_t c_s, int32_t heads) {
  if (n <= 0 || c_s <= 0 || heads <= 0) return 0;
  return standalone_plan(n, c_s, heads).total + 1024;  // the workspace may start anywhere: aligned up inside
}

extern "C" int b200tri_attention_pair_bias(const b200tri_attention_pair_bias_args* a, b200tri_stream_t stream_) {
  using namespace b200;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "attention pair bias: null args");
  B200_REQUIRE(a->s && a->z && a->mask && a->out && a->proj_q && a->proj_q_bias && a->proj_k && a->proj_v && a->proj_g &&
                   a->proj_z_norm_scale && a->proj_z_norm_bias && a->proj_z && a->proj_o,
               B200TRI_ERR_INVALID, "attention pair bias: null pointer argument");
  B200_REQUIRE(a->n > 0, B200TRI_ERR_INVALID, "attention pair bias: n must be positive");
  B200_REQUIRE(a->c_z == C_Z, B200TRI_ERR_UNSUPPORTED, "attention pair bias: built for c_z = 128 (got %d)", a->c_z);
  B200_REQUIRE(a->heads >= 1 && a->heads <= MAX_HEADS && a->c_s == a->heads * HD, B200TRI_ERR_UNSUPPORTED,
               "attention pair bias: built for up to 16 heads of width 24 (got c_s %d, %d heads)", a->c_s, a->heads);
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a->z) & 15) == 0, B200TRI_ERR_INVALID,
               "attention pair bias: z must be 16-byte aligned");
  const size_t need = b200tri_attention_pair_bias_workspace_bytes(a->n, a->c_s, a->heads);
  B200_REQUIRE(a->workspace && a->workspace_bytes >= need, B200TRI_ERR_WORKSPACE,
               "attention pair bias: workspace of %zu bytes needed", need);
  const StandalonePlan pl = standalone_plan(a->n, a->c_s, a->heads);
  uint8_t* ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(a->workspace) + 1023) & ~uintptr_t(1023));
  __nv_bfloat16* xq = reinterpret_cast<__nv_bfloat16*>(ws + pl.xq);
  __nv_bfloat16* xk = xq;
  float* partial = reinterpret_cast<float*>(ws + pl.partial);
  RowArgs row = {};
  row.rows = a->n;
  row.c = a->c_s;
  row.base = static_cast<const float*>(a->s);
  row.pieces = xq;
  int rc = launch_row_norm(row, stream, false);
  if (rc) return rc;
  if (a->k_in && a->k_in != a->s) {
    xk = reinterpret_cast<__nv_bfloat16*>(ws + pl.xk);
    row.base = static_cast<const float*>(a->k_in);
    row.pieces = xk;
    if ((rc = launch_row_norm(row, stream, false))) return rc;
  }
  int splits = 1;
  if ((rc = single_project(a, xq, xk, ws + pl.work, stream)) || (rc = single_pair_bias(a, ws + pl.work, stream, true)) ||
      (rc = single_attend(a, ws + pl.work, partial, &splits, stream, true)))
    return rc;
  row.base = nullptr;
  row.partial = partial;
  row.splits = splits;
  row.pieces = nullptr;
  row.sum_out = static_cast<float*>(a->out);
  return launch_row_norm(row, stream, true);
}
