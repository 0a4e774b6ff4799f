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
// The only part that scales with N^2 * c_z is the pair-bias pass over z
// (pair_bias_kernel, HBM-bound: 256 B read and 4 * heads B written per pair); the
// token attention itself is N^2 * c_s work (14 GFLOP at N = 3072) and runs on the
// fp32 pipes: at 16 heads x 24 channels it is far too small to be worth tensor-core
// tiles, and its operands are fp32.
#include "host.cuh"
#include "single.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int C_Z = 128;
constexpr int MAX_HEADS = 16;
constexpr int HD = 24;  // head width the token-attention kernel is built for

// ---------------------------------------------------------------- pair bias
// One thread per pair, 128 pairs per tile. With gamma folded into the projection,
//   bias_h = rstd * (sum_c x_c W'[c][h] - mean * sum_c W'[c][h]) + sum_c beta_c W[c][h],
// so the normalised row is never formed: one pass for the mean, one for the variance
// (two-pass, as the reference computes it), one pass of heads FMAs per channel. The tile is
// loaded with coalesced 16-byte loads into shared memory (16-byte chunks XOR-swizzled by the
// pair index, so that neither the row-major stores nor the thread-per-row reads conflict)
// and every pass reads it from there: the row never has to live in registers, and the
// projection runs two heads per instruction (fma.f32x2).
__global__ void __launch_bounds__(128, 4)
pair_bias_kernel(const __nv_bfloat16* __restrict__ z, long long n_pairs, int n, int ld, int heads,
                 const __nv_bfloat16* __restrict__ ln_scale, const __nv_bfloat16* __restrict__ ln_bias,
                 const __nv_bfloat16* __restrict__ wz, float eps, float* __restrict__ bias) {
  __shared__ __align__(16) float w[C_Z][MAX_HEADS];  // gamma_c * Wz[c][h]
  __shared__ float sw[MAX_HEADS], bw[MAX_HEADS];
  __shared__ __align__(16) uint4 tile_s[128 * 16];   // 128 pairs x 16 chunks of 8 channels
  for (int idx = threadIdx.x; idx < C_Z * MAX_HEADS; idx += blockDim.x) {
    const int c = idx / MAX_HEADS, h = idx % MAX_HEADS;
    w[c][h] = h < heads ? __bfloat162float(ln_scale[c]) * __bfloat162float(wz[c * heads + h]) : 0.f;
  }
  __syncthreads();
  if (threadIdx.x < MAX_HEADS) {
    const int h = threadIdx.x;
    float a = 0.f, b = 0.f;
    for (int c = 0; c < C_Z; ++c) {
      a += w[c][h];
      if (h < heads) b += __bfloat162float(ln_bias[c]) * __bfloat162float(wz[c * heads + h]);
    }
    sw[h] = a;
    bw[h] = b;
  }
  __syncthreads();
  const long long tiles = (n_pairs + 127) / 128;
  const int p = threadIdx.x, key = p & 15;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long base = tile * 128;
    const long long left = n_pairs - base;  // pairs of this tile that exist (>= 1)
    const uint4* src = reinterpret_cast<const uint4*>(z + base * C_Z);
#pragma unroll 8
    for (int it = 0; it < 16; ++it) {
      const int idx = it * 128 + p;  // chunk idx of the tile: pair idx / 16, chunk idx % 16
      const int pr = idx >> 4, ch = idx & 15;
      const uint4 v = pr < left ? src[idx] : make_uint4(0u, 0u, 0u, 0u);
      tile_s[pr * 16 + (ch ^ (pr & 15))] = v;
    }
    __syncthreads();
    const uint4* row = tile_s + p * 16;
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 v = row[c ^ key];
      const uint32_t x4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) s4[e] += bf16_lo(x4[e]) + bf16_hi(x4[e]);
    }
    const float mean = ((s4[0] + s4[1]) + (s4[2] + s4[3])) * (1.0f / C_Z);
    float q4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 v = row[c ^ key];
      const uint32_t x4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float a = bf16_lo(x4[e]) - mean, b = bf16_hi(x4[e]) - mean;
        q4[e] = fmaf(a, a, q4[e]);
        q4[e] = fmaf(b, b, q4[e]);
      }
    }
    const float rstd = rsqrtf(((q4[0] + q4[1]) + (q4[2] + q4[3])) * (1.0f / C_Z) + eps);
    float2 acc[MAX_HEADS / 2];
#pragma unroll
    for (int h = 0; h < MAX_HEADS / 2; ++h) acc[h] = make_float2(0.f, 0.f);
#pragma unroll 2
    for (int c = 0; c < 16; ++c) {
      const uint4 v = row[c ^ key];
      const uint32_t x4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int ch = 8 * c + 2 * e;  // channels ch (low half) and ch + 1 (high half)
        const float a = bf16_lo(x4[e]), b = bf16_hi(x4[e]);
        const float2 a2 = make_float2(a, a), b2 = make_float2(b, b);
        const float4* wa = reinterpret_cast<const float4*>(w[ch]);
        const float4* wb = reinterpret_cast<const float4*>(w[ch + 1]);
#pragma unroll
        for (int h4 = 0; h4 < MAX_HEADS / 4; ++h4) {
          const float4 fa = wa[h4], fb = wb[h4];
          acc[2 * h4 + 0] = __ffma2_rn(b2, make_float2(fb.x, fb.y), __ffma2_rn(a2, make_float2(fa.x, fa.y), acc[2 * h4 + 0]));
          acc[2 * h4 + 1] = __ffma2_rn(b2, make_float2(fb.z, fb.w), __ffma2_rn(a2, make_float2(fa.z, fa.w), acc[2 * h4 + 1]));
        }
      }
    }
    const long long pair = base + p;
    if (pair < n_pairs) {
      const long long i = pair / n, j = pair % n;
#pragma unroll
      for (int h = 0; h < MAX_HEADS; ++h)
        if (h < heads)
          bias[(static_cast<long long>(h) * n + i) * ld + j] = rstd * ((h & 1 ? acc[h >> 1].y : acc[h >> 1].x) - mean * sw[h]) + bw[h];
    }
    __syncthreads();  // the tile is overwritten by the next round's loads
  }
}

// ------------------------------------------------------------------ row kernels
// See launch_row_norm. One warp per row, the row in registers (up to 12 values per lane).
constexpr int ROW_VALUES = MAX_HEADS * HD / 32;
__global__ void __launch_bounds__(128) row_norm_kernel(const RowArgs a) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= a.rows) return;
  const long long off = static_cast<long long>(row) * a.c;
  const bool keep = a.row_mask == nullptr || a.row_mask[row] != 0.f;
  float v[ROW_VALUES];
  float s = 0.f;
#pragma unroll
  for (int e = 0; e < ROW_VALUES; ++e) {
    const int i = lane + 32 * e;
    v[e] = 0.f;
    if (i >= a.c || !keep) continue;
    if (a.partial) {
      float u = 0.f;
      for (int p = 0; p < a.splits; ++p) u += a.partial[static_cast<long long>(p) * a.rows * a.c + off + i];
      v[e] = u;
    }
    if (a.base) v[e] = a.base[off + i] + v[e];
    s += v[e];
  }
  if (a.sum_out) {
#pragma unroll
    for (int e = 0; e < ROW_VALUES; ++e)
      if (lane + 32 * e < a.c) a.sum_out[off + lane + 32 * e] = v[e];
  }
  if (!a.pieces) return;
  if (a.scale) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    const float mean = s / a.c;
    float q = 0.f;
#pragma unroll
    for (int e = 0; e < ROW_VALUES; ++e)
      if (lane + 32 * e < a.c) q += (v[e] - mean) * (v[e] - mean);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) q += __shfl_xor_sync(0xffffffffu, q, d);
    const float rstd = 1.0f / sqrtf(q / a.c + a.eps);
    const __nv_bfloat16* scale = static_cast<const __nv_bfloat16*>(a.scale);
    const __nv_bfloat16* bias = static_cast<const __nv_bfloat16*>(a.bias);
#pragma unroll
    for (int e = 0; e < ROW_VALUES; ++e) {
      const int i = lane + 32 * e;
      if (i < a.c) v[e] = (v[e] - mean) * rstd * __bfloat162float(scale[i]) + __bfloat162float(bias[i]);
    }
  }
  const long long plane = static_cast<long long>(a.rows) * a.c;
#pragma unroll
  for (int e = 0; e < ROW_VALUES; ++e) {
    const int i = lane + 32 * e;
    if (i >= a.c) continue;
    __nv_bfloat16* dst = a.pieces + off + i;
    split3(v[e], dst[0], dst[plane], dst[2 * plane]);
  }
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
// float32 activations (three pieces) x bf16 weights as stored. The old CUDA-core kernel took
// 116 us for 128 x 384 x 384 (six blocks on the whole chip, 24 dependent k steps of scalar
// loads); the products of a block are 0.6-15 GFLOP, so what bounds them at every size is
// latency: many small tiles, K split until the tiles cover the SMs.
//
// [q | k | v | g] in one launch: column tiles of 64 walk the four weights in turn.
struct QkvgPolicy {
  static constexpr int BN = 64, PA = 3, PB = 1, NSEG = 1, NMAIN = 3;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = 8, CTAS = 1;
  struct Params {
    int rows, c, tiles_per_w, first_w;
    const __nv_bfloat16* q_bias;
    float* out[4];
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
                                  int col0, int col1, int lane) {
    const int row = m_tile * GEMM_BM + quarter * 32 + lane;
    const int which = p.first_w + n_tile / p.tiles_per_w;
#pragma unroll 1
    for (int col = col0; col < col1; col += 16) {
    float r[16];
    acc.load(0, col, r);
    if (row >= p.rows) continue;
    const int c0 = n_tile % p.tiles_per_w * BN + col;
    float* dst = p.out[which] + static_cast<long long>(row) * p.c + c0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v[4];
      if (c0 + 4 * q >= p.c) break;  // c is a multiple of 8
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[e] = r[4 * q + e];
        if (which == 0) v[e] += __bfloat162float(p.q_bias[c0 + 4 * q + e]);
        if (which == 3) v[e] = 1.0f / (1.0f + expf(-v[e]));
      }
      *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(v[0], v[1], v[2], v[3]);
    }
    }
  }
};

// float32 partial sums, one plane per K split.
struct PartialPolicy {
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
                                  int quarter, int col0, int col1, int lane) {
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
struct SwigluPolicy {
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
                                  int col0, int col1, int lane) {
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

// --------------------------------------------------------- token attention
// One thread per (query i, head h); keys in tiles of 32 staged in shared memory.
// Online softmax in fp32; scores = q.k / sqrt(d) + bias + (1 - mask) * -inf, added in
// that order like the reference (attention.py:134-136).
constexpr int TQ = 64;  // queries per block
constexpr int TK = 32;  // keys per tile

__global__ void __launch_bounds__(TQ)
token_attention_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                       const float* __restrict__ gate, const float* __restrict__ bias, const float* __restrict__ mask, int n,
                       int n_keys, int ld, int c_s, float inf, __nv_bfloat16* __restrict__ out) {
  __shared__ float ks[TK][HD], vs[TK][HD], ms[TK];
  const int h = blockIdx.y;
  const int i = blockIdx.x * TQ + threadIdx.x;
  const bool live = i < n;
  const float inv_scale = 1.0f / sqrtf(static_cast<float>(HD));
  float qr[HD], acc[HD];
#pragma unroll
  for (int d = 0; d < HD; ++d) {
    qr[d] = live ? q[static_cast<long long>(i) * c_s + h * HD + d] : 0.f;
    acc[d] = 0.f;
  }
  float m_run = -INFINITY, l_run = 0.f;
  const float* brow = bias + (static_cast<long long>(h) * n + (live ? i : 0)) * ld;
  for (int j0 = 0; j0 < n_keys; j0 += TK) {
    __syncthreads();
    for (int idx = threadIdx.x; idx < TK * HD; idx += TQ) {
      const int r = idx / HD, d = idx % HD;
      const int j = j0 + r;
      ks[r][d] = j < n_keys ? k[static_cast<long long>(j) * c_s + h * HD + d] : 0.f;
      vs[r][d] = j < n_keys ? v[static_cast<long long>(j) * c_s + h * HD + d] : 0.f;
    }
    if (threadIdx.x < TK) {
      const int j = j0 + threadIdx.x;
      ms[threadIdx.x] = j < n_keys ? (1.0f - mask[j]) * -inf : -INFINITY;  // keys past the end: no weight
    }
    __syncthreads();
    float sc[TK];
    float mx = m_run;
#pragma unroll
    for (int r = 0; r < TK; ++r) {
      float dot = 0.f;
#pragma unroll
      for (int d = 0; d < HD; ++d) dot = fmaf(qr[d], ks[r][d], dot);
      const float b = (j0 + r < n_keys) ? brow[j0 + r] : 0.f;
      sc[r] = (dot * inv_scale + b) + ms[r];
      mx = fmaxf(mx, sc[r]);
    }
    const float alpha = __expf(m_run - mx);  // 0 on the first tile
    l_run *= alpha;
#pragma unroll
    for (int d = 0; d < HD; ++d) acc[d] *= alpha;
#pragma unroll
    for (int r = 0; r < TK; ++r) {
      const float pr = __expf(sc[r] - mx);
      l_run += pr;
#pragma unroll
      for (int d = 0; d < HD; ++d) acc[d] = fmaf(pr, vs[r][d], acc[d]);
    }
    m_run = mx;
  }
  if (live) {
    const float inv = 1.0f / l_run;
    const long long off = static_cast<long long>(i) * c_s + h * HD, plane = static_cast<long long>(n) * c_s;
#pragma unroll
    for (int d = 0; d < HD; ++d) {  // gated, as the pieces the output projection reads
      __nv_bfloat16* dst = out + off + d;
      split3(acc[d] * inv * gate[off + d], dst[0], dst[plane], dst[2 * plane]);
    }
  }
}

}  // namespace

int launch_row_norm(const RowArgs& a, cudaStream_t stream, bool pdl) {
  return launch(row_norm_kernel, dim3((a.rows + 3) / 4), dim3(128), 0, stream, pdl, a);
}

// Enough splits that the tiles cover the SMs, at least two k steps each, none of them empty.
int single_splits(int tiles, int kb) {
  int s = 148 / (tiles > 0 ? tiles : 1);
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
  w.q = take(act * 4);
  w.k = take(act * 4);
  w.v = take(act * 4);
  w.g = take(act * 4);
  w.bias = take(static_cast<size_t>(heads) * n * round_up(n, 4) * 4);
  w.ao = take(act * 2 * 3);
  for (size_t& off : w.w) off = take(tma_weight_bytes(c_s, c_s));
  w.total = c.total();
  return w;
}

int single_attention(const b200tri_attention_pair_bias_args* a, const __nv_bfloat16* xq, const __nv_bfloat16* xk,
                     uint8_t* work, float* partial, int* splits, cudaStream_t stream) {
  const int n = a->n, c_s = a->c_s, heads = a->heads, ld = round_up(n, 4);
  const SingleAttentionWork off = single_attention_work(n, c_s, heads);
  float* out[4] = {reinterpret_cast<float*>(work + off.q), reinterpret_cast<float*>(work + off.k),
                   reinterpret_cast<float*>(work + off.v), reinterpret_cast<float*>(work + off.g)};
  float* bias = reinterpret_cast<float*>(work + off.bias);
  __nv_bfloat16* ao = reinterpret_cast<__nv_bfloat16*>(work + off.ao);
  auto bf = [](const void* p) { return static_cast<const __nv_bfloat16*>(p); };

  // q, k, v, g. With separate key-side rows: k, v from those in a launch of their own
  // (weights in the order q, g | k, v then).
  const bool same = xq == xk;
  const void* w_same[4] = {a->proj_q, a->proj_k, a->proj_v, a->proj_g};
  GemmMaps maps = {};
  bool direct = true;
  int rc;
  for (int i = 0; i < 4; ++i) {
    const void* wp;
    long long pitch;
    if ((rc = tma_weight(w_same[i], c_s, c_s, work + off.w[i], stream, &wp, &pitch))) return rc;
    if ((rc = gemm_map_mnmajor(&maps.b[i], wp, c_s, c_s, pitch))) return rc;
    direct = direct && wp == w_same[i];
  }
  const int per_w = (c_s + QkvgPolicy::BN - 1) / QkvgPolicy::BN;
  QkvgPolicy::Params ep = {n, c_s, per_w, 0, bf(a->proj_q_bias), {out[0], out[1], out[2], out[3]}};
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
  {
    TimedLaunch timed(K_PAIR_BIAS, stream);
    const long long n_pairs = static_cast<long long>(n) * n;
    const long long tiles = (n_pairs + 127) / 128;
    const long long blocks = tiles < 16LL * sm_count() ? tiles : 16LL * sm_count();
    count_launch();
    pair_bias_kernel<<<static_cast<unsigned>(blocks), 128, 0, stream>>>(bf(a->z), n_pairs, n, ld, heads,
                                                                       bf(a->proj_z_norm_scale), bf(a->proj_z_norm_bias),
                                                                       bf(a->proj_z), a->eps, bias);
    B200_CUDA_OK(cudaGetLastError());
  }
  count_launch();
  token_attention_kernel<<<dim3((n + TQ - 1) / TQ, heads), TQ, 0, stream>>>(
      out[0], out[1], out[2], out[3], bias, static_cast<const float*>(a->mask), n, n, ld, c_s, a->inf, ao);
  B200_CUDA_OK(cudaGetLastError());
  return launch_linear_partial(ao, c_s, n, c_s, a->proj_o, c_s, work + off.w[4], partial, splits, stream, false);
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
  if ((rc = single_attention(a, xq, xk, ws + pl.work, partial, &splits, stream))) return rc;
  row.base = nullptr;
  row.partial = partial;
  row.splits = splits;
  row.pieces = nullptr;
  row.sum_out = static_cast<float*>(a->out);
  return launch_row_norm(row, stream, true);
}
