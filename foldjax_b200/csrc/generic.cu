// The two triangle ops for every shape and element type the fused 128-channel bf16 kernels do
// not cover:
//
//  * the float32 trunk of the reference at the specialised shape (a correctness mode with a
//    1e-4 bar: triangle_multiplication_forward's default contraction precision is float32,
//    src/foldjax/models/boltz2/models/triangle/triangle.py:95-96);
//  * other call sites of the same ops - the template stacks (c_z = 64 with c_hidden = 128,
//    which the cuEquivariance kernel rejects, src/foldjax/models/protenix/models/triangle/
//    triangle.py:131-137), the 384-channel / 12-head structural refiner
//    (src/foldjax/models/opendde/structural_refiner.py:62), other head counts and widths -
//    in bf16 or float32.
//
// Structure: every product runs on the tensor cores (gemm.cuh), with bf16 operands as they are
// and float32 operands as three bf16 pieces; gates, masks, rounding and layout changes sit in
// the products' epilogues, so that a multiplicative update is five launches
//   layer norm -> [gate|value] product -> contraction -> layer norm -> output product
// and an attention five
//   layer norm -> q, k, v, bias product -> core -> gate product -> output product
// (plus one that splits or pads weights where they cannot be read as stored). The layer norms
// are CUDA-core kernels. The four updates of a 256-token 384-channel refiner block take 1.05 ms and
// those of four 200-token templates 0.54 (26.2 and 6.9 with the products on the CUDA cores). What the
// threads of an epilogue move, each along a row of its own, goes 32 bytes at a time: with 16 those
// stacks took 1.29 and 0.80 ms and a 256-token float32 stack 1.01 instead of 0.91.
//
// With a bf16 trunk every point where the reference's bf16 arrays round (after each matmul,
// the sigmoid, each elementwise product or sum, the two steps of the layer-norm affine,
// q / sqrt(d), the contraction and the attention output) is rounded here too (`Rb`), so the
// results follow the same recipe as the specialised kernels; with float32 nothing is rounded.
#include <cuda_bf16.h>
#include <math.h>

#include <type_traits>

#include <string.h>

#include "att_split.cuh"
#include "gemm.cuh"
#include "host.cuh"
#include "tc.cuh"

namespace b200 {
namespace {

// Rounding policy of the trunk dtype.
template <bool BF>
struct Rb {
  static __device__ __forceinline__ float r(float v) { return BF ? round_bf16(v) : v; }
};

__device__ __forceinline__ float sigmoid_exact(float x) { return 1.0f / (1.0f + expf(-x)); }

// Two neighbouring values as PIECES packed words, `plane` elements apart (dst 4-byte aligned).
template <int PIECES>
__device__ __forceinline__ void store_pair(__nv_bfloat16* dst, long long plane, float a, float b) {
  if (PIECES == 1) {
    *reinterpret_cast<uint32_t*>(dst) = pack_bf16x2(a, b);
  } else {
    uint32_t hi, mid, lo;
    split3x2(a, b, hi, mid, lo);
    *reinterpret_cast<uint32_t*>(dst) = hi;
    *reinterpret_cast<uint32_t*>(dst + plane) = mid;
    *reinterpret_cast<uint32_t*>(dst + 2 * plane) = lo;
  }
}
// Eight neighbouring values the same way (dst 16-byte aligned).
template <int PIECES>
__device__ __forceinline__ void store_eight(__nv_bfloat16* dst, long long plane, const float* v) {
  uint32_t w[3][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (PIECES == 1) {
      w[0][e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
    } else {
      split3x2(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
    }
  }
#pragma unroll
  for (int q = 0; q < PIECES; ++q) *reinterpret_cast<uint4*>(dst + q * plane) = make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]);
}
// Sixteen of them (dst and plane on 32-byte boundaries), a sector per piece.
template <int PIECES>
__device__ __forceinline__ void store_sixteen(__nv_bfloat16* dst, long long plane, const float* v) {
  uint32_t w[3][8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (PIECES == 1) {
      w[0][e] = pack_bf16x2(v[2 * e], v[2 * e + 1]);
    } else {
      split3x2(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
    }
  }
#pragma unroll
  for (int q = 0; q < PIECES; ++q)
    store_sector(dst + q * plane, make_uint4(w[q][0], w[q][1], w[q][2], w[q][3]), make_uint4(w[q][4], w[q][5], w[q][6], w[q][7]));
}
// Eight neighbouring values to the caller's tensor, with the caller's residual added (one more
// rounding of the trunk dtype).
template <bool BF, typename O>
__device__ __forceinline__ void store_out(O* dst, const O* res, float* v, bool aligned, bool sectors) {
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = Rb<BF>::r(v[e]);
  if constexpr (!BF) {
    if (sectors) {
      uint4 a, b;
      if (res) {
        load_sector(res, a, b);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(w[e]) + v[e];
      }
      a = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
      b = make_uint4(__float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7]));
      store_sector(dst, a, b);
      return;
    }
  }
  if (aligned) {
    constexpr int W = 8 * sizeof(O) / 16;
    uint4 raw[W];
    O* o = reinterpret_cast<O*>(raw);
    if (res) {
#pragma unroll
      for (int w = 0; w < W; ++w) raw[w] = reinterpret_cast<const uint4*>(res)[w];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = Rb<BF>::r(static_cast<float>(o[e]) + v[e]);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = static_cast<O>(v[e]);
#pragma unroll
    for (int w = 0; w < W; ++w) reinterpret_cast<uint4*>(dst)[w] = raw[w];
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) dst[e] = static_cast<O>(res ? Rb<BF>::r(static_cast<float>(res[e]) + v[e]) : v[e]);
  }
}

// -------------------------------------------------------------------------- weights
// dst[piece][k][ld] = pieces of src[k][n], padding columns zero: float32 weights, and bf16 ones
// whose pitch or address TMA cannot take.
struct WeightJob {
  const void* src;
  __nv_bfloat16* dst;
  int k, n, ld;
};
struct WeightJobs {
  WeightJob job[6];
};
template <bool BF>
__global__ void weight_kernel(const WeightJobs jobs) {
  pdl_wait();
  pdl_trigger();
  const WeightJob j = jobs.job[blockIdx.y];
  const long long total = static_cast<long long>(j.k) * j.ld;
  for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int r = static_cast<int>(idx / j.ld), c = static_cast<int>(idx % j.ld);
    const long long at = static_cast<long long>(r) * j.n + c;
    if (BF) {
      j.dst[idx] = c < j.n ? static_cast<const __nv_bfloat16*>(j.src)[at] : __float2bfloat16_rn(0.f);
    } else {
      split3(c < j.n ? static_cast<const float*>(j.src)[at] : 0.f, j.dst[idx], j.dst[total + idx], j.dst[2 * total + idx]);
    }
  }
}

// ------------------------------------------------------------------ layer norm + gather
// Means over c channels. The product with the rounded reciprocal alone is off to the same side in
// every row unless c is a power of two: where the mean is 5000 deviations the float32 attention of 384
// channels was 5.1e-4 from float64, 7 times what it is with quotients. One correction by the residual
// (Markstein, 1990) gives the rounded quotient; a division costs 1 % of a template stack.
struct Channels {
  float c, inv;
  __device__ explicit Channels(int n) : c(static_cast<float>(n)), inv(1.0f / c) {}
  __device__ __forceinline__ float mean(float sum) const {
    const float q = sum * inv;
    return fmaf(fmaf(-q, c, sum), inv, q);
  }
};

// xn[piece][(b, o, t)][:] = LN(x[b][o * xs_o + t * xs_i + :]). A warp takes a few successive t of
// one row, each in the registers of a group of lanes, so that the loads of all of them are in
// flight together. Optionally the pair's mask bias of the attention core, mb[(b, o)][t] (the
// pitch padding with the last pair of a row).
// Bound: HBM / L2 traffic. The grid is (t, o, b): no divisions.
struct LnArgs {
  const void* x;
  long long xs_b, xs_o, xs_i;
  int batch, n, c;
  const void* scale;
  const void* bias;
  float eps;
  __nv_bfloat16* xn;
  bool aligned, aligned_params;  // x, and scale and bias, start on a 16-byte boundary
  float* mb;     // or null
  const float* mask;
  long long ms_b, ms_o, ms_i;
  float inf;
  int mb_ld;
};
constexpr int LN_WARPS = 8;
// Eight neighbouring values of a row as floats (p 16-byte aligned, or anywhere).
template <bool BF, typename X>
__device__ __forceinline__ void load_eight(const X* p, bool aligned, float (&v)[8]) {
  if (aligned) {
    uint4 raw[BF ? 1 : 2];
#pragma unroll
    for (int w = 0; w < (BF ? 1 : 2); ++w) raw[w] = reinterpret_cast<const uint4*>(p)[w];
    const X* x = reinterpret_cast<const X*>(raw);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = static_cast<float>(x[e]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = static_cast<float>(p[e]);
  }
}
// The same as they are, of a bf16 row.
__device__ __forceinline__ uint4 eight_raw(const __nv_bfloat16* p, bool aligned) {
  if (aligned) return *reinterpret_cast<const uint4*>(p);
  const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
  return make_uint4(u[0] | (static_cast<uint32_t>(u[1]) << 16), u[2] | (static_cast<uint32_t>(u[3]) << 16),
                    u[4] | (static_cast<uint32_t>(u[5]) << 16), u[6] | (static_cast<uint32_t>(u[7]) << 16));
}
// bf16(bf16(bf16(d * rstd) * scale) + bias) of two deviations from the mean. Value by value, with conversions to
// and from float32 at every rounding, the layer norms issued 35 to 46 instructions per value and nothing
// else bounded them: 160 000 rows of 64 channels took 17 us, their channel-major form of 128 channels 40.
__device__ __forceinline__ uint32_t affine_bf16x2(float2 d, float2 rstd, uint32_t scale, uint32_t bias) {
  const float2 t = __fmul2_rn(d, rstd);
  return bf16x2_add(bf16x2_mul(pack_bf16x2(t.x, t.y), scale), bias);
}
// L neighbouring lanes per row, K chunks of eight channels per lane, R rows of a lane group in
// flight. (With a row per warp and two channels per lane the 64-channel case took 24 us for
// 160 000 rows, half of it the five exchanges of every sum; three are left.)
template <bool BF, int L, int K, int R>
__global__ void __launch_bounds__(LN_WARPS * 32) ln_gather_kernel(const LnArgs a) {
  using X = typename std::conditional<BF, __nv_bfloat16, float>::type;
  constexpr int GROUPS = 32 / L, ROWS = GROUPS * R;  // rows of a warp
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int t0 = (blockIdx.x * LN_WARPS + (threadIdx.x >> 5)) * ROWS, o = blockIdx.y, b = blockIdx.z;
  if (t0 >= a.n) return;
  const int bo = b * a.n + o;
  if (a.mb) {
    float* row = a.mb + static_cast<long long>(bo) * a.mb_ld;
    if (lane < ROWS && t0 + lane < a.n)
      row[t0 + lane] = a.mask ? fmaxf(a.inf * (a.mask[b * a.ms_b + o * a.ms_o + (t0 + lane) * a.ms_i] - 1.0f), SPLIT_MASK_MIN) : 0.f;
    if (t0 + ROWS >= a.n)
      for (int e = a.n + lane; e < a.mb_ld; e += 32) row[e] = SPLIT_MASK_PAD;
  }
  const int c0 = (lane % L) * 8, t_lane = t0 + lane / L;  // the lane's rows are t_lane + GROUPS * r
  const X* src = static_cast<const X*>(a.x) + b * a.xs_b + o * a.xs_o;
  float v[R][K][8];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const X* row = src + min(t_lane + GROUPS * r, a.n - 1) * a.xs_i;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int c = c0 + k * L * 8;
      if (c < a.c) {
        load_eight<BF>(row + c, a.aligned, v[r][k]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[r][k][e] = 0.f;
      }
    }
  }
  const Channels chans(a.c);
  float s[R], q[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    s[r] = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int e = 0; e < 8; e += 2) s[r] += v[r][k][e] + v[r][k][e + 1];
  }
#pragma unroll
  for (int d = L / 2; d > 0; d >>= 1)
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], d);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    s[r] = chans.mean(s[r]);
    q[r] = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (c0 + k * L * 8 < a.c)
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const float2 d = __fadd2_rn(make_float2(v[r][k][e], v[r][k][e + 1]), make_float2(-s[r], -s[r]));
          q[r] = fmaf(d.y, d.y, fmaf(d.x, d.x, q[r]));
          if constexpr (BF) {  // the deviations take the values' place (template stack 546.0 -> 542.4 us)
            v[r][k][e] = d.x;
            v[r][k][e + 1] = d.y;
          }
        }
  }
#pragma unroll
  for (int d = L / 2; d > 0; d >>= 1)
#pragma unroll
    for (int r = 0; r < R; ++r) q[r] += __shfl_xor_sync(0xffffffffu, q[r], d);
#pragma unroll
  for (int r = 0; r < R; ++r) q[r] = 1.0f / sqrtf(chans.mean(q[r]) + a.eps);
  const long long plane = static_cast<long long>(a.batch) * a.n * a.n * a.c;
  __nv_bfloat16* dst = a.xn + (static_cast<long long>(bo) * a.n + t_lane) * a.c;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int c = c0 + k * L * 8;
    if (c >= a.c) continue;
    if constexpr (BF) {  // cast before the affine step, whose two roundings are those of packed bf16 operations
      const uint4 g4 = eight_raw(static_cast<const __nv_bfloat16*>(a.scale) + c, a.aligned_params);
      const uint4 h4 = eight_raw(static_cast<const __nv_bfloat16*>(a.bias) + c, a.aligned_params);
      const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w}, h[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (t_lane + GROUPS * r >= a.n) break;
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          w[e] = affine_bf16x2(make_float2(v[r][k][2 * e], v[r][k][2 * e + 1]), make_float2(q[r], q[r]), g[e], h[e]);
        *reinterpret_cast<uint4*>(dst + GROUPS * r * a.c + c) = make_uint4(w[0], w[1], w[2], w[3]);
      }
      continue;
    }
    float g[8], h[8];
    load_eight<BF>(static_cast<const X*>(a.scale) + c, a.aligned_params, g);
    load_eight<BF>(static_cast<const X*>(a.bias) + c, a.aligned_params, h);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (t_lane + GROUPS * r >= a.n) break;
      float u[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)  // cast before the affine step
        u[e] = Rb<BF>::r(Rb<BF>::r(Rb<BF>::r((v[r][k][e] - s[r]) * q[r]) * g[e]) + h[e]);
      store_eight<BF ? 1 : 3>(dst + GROUPS * r * a.c + c, plane, u);
    }
  }
}

template <bool BF>
int launch_ln_gather(LnArgs a, cudaStream_t stream, bool pdl) {
  a.aligned = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0;  // (rows are multiples of eight values apart)
  a.aligned_params = ((reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.bias)) & 15) == 0;
  auto go = [&](auto kernel, int rows) {
    const int per_block = LN_WARPS * rows;
    const dim3 grid((a.n + per_block - 1) / per_block, static_cast<unsigned>(a.n), static_cast<unsigned>(a.batch));
    return launch(kernel, grid, dim3(LN_WARPS * 32), 0, stream, pdl, a);
  };
  if (a.c <= 64) return go(ln_gather_kernel<BF, 8, 1, 2>, 8);
  if (a.c <= 128) return go(ln_gather_kernel<BF, 16, 1, 2>, 4);
  if (a.c <= 256) return go(ln_gather_kernel<BF, 32, 1, 2>, 2);
  if (a.c <= 384) return go(ln_gather_kernel<BF, 16, 3, 1>, 2);
  return go(ln_gather_kernel<BF, 32, 4, 1>, 1);
}

// ------------------------------------------------------------ tri-mult: LN of the contraction
// tn[piece][(b, i, j)][:] = LN_out(t[b][:, i, j]) with t channel-major [b * c_h + channel][n][ld],
// rounded to the trunk dtype before the layer norm (triangle.py:124-126). One block = 128 bytes
// of neighbouring j of a row (64 in bf16, 32 in float32) with all their channels in shared
// memory. A lane owns one word of that row - two j in bf16, one in float32 - and a warp an
// eighth of the channels, so that the statistics are plain sums per lane (one exchange of eight
// partial sums each) and nothing is shuffled: 40 instructions per pair where one warp per pair
// took 209. Eight neighbouring channels per lane are 16 bytes; in bf16, up to 64 * G channels, they
// are put together in shared memory (over the values, when all have been read) and leave as one
// contiguous run: stored by the lanes themselves they went to 64 rows, half a sector each. In
// float32, up to 384 channels, the three pieces have a place of their own behind the values (G = 1). That
// leaves 3 / 2 / 1 blocks to an SM at 192 / 256 / 384 channels. The whole multiplication staged and not,
// us: 128 channels, 256 tokens 181 / 192; 192, 96 and 256 tokens 110 / 128 and 415 / 429; 256, 96 and 256 tokens
// 140 / 154 and 619 / 614; 320, 96 and 256 tokens 198 / 225 and 890 / 906; 384, 96 and 256 tokens 252 / 269 and
// 1202 / 1175 (of the latter 270 and 1250 with 16-byte accesses).
constexpr int LNT_WARPS = 8;
template <bool BF>
constexpr int lnt_j() {
  return BF ? 64 : 32;
}
inline int lnt_smem(int c_h) { return c_h * 128 + 2 * LNT_WARPS * 64 * 4 + c_h * 8; }
template <bool BF, int G>
__global__ void __launch_bounds__(LNT_WARPS * 32)
ln_channel_major_kernel(const void* __restrict__ t_, int n, int ld, int c_h, const void* __restrict__ scale_,
                        const void* __restrict__ bias_, float eps, long long pairs, __nv_bfloat16* __restrict__ tn) {
  using X = typename std::conditional<BF, __nv_bfloat16, float>::type;
  constexpr int JT = lnt_j<BF>(), JL = JT / 32;  // j of a block, of a lane
  extern __shared__ uint32_t tile[];             // [c_h][32 words], then the partial sums, then scale and bias
  float* part = reinterpret_cast<float*>(tile + (c_h + 63) / 64 * 64 * 32);
  uint2* affine = reinterpret_cast<uint2*>(part + 2 * LNT_WARPS * 64);  // bf16: each twice in a word
  pdl_wait();
  pdl_trigger();
  if constexpr (BF)
    for (int c = threadIdx.x; c < c_h; c += LNT_WARPS * 32) {
      const uint32_t sc = static_cast<const unsigned short*>(scale_)[c], bi = static_cast<const unsigned short*>(bias_)[c];
      affine[c] = make_uint2(sc | sc << 16, bi | bi << 16);
    }
  const int i = blockIdx.y, b = blockIdx.z, j0 = blockIdx.x * JT;
  const X* src = static_cast<const X*>(t_) + (static_cast<long long>(b) * c_h * n + i) * ld + j0;
  const long long chan = static_cast<long long>(n) * ld;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // groups of eight channels, dealt to the warps in turn
  const int groups = c_h / 8;
  auto value = [&](uint32_t w, int u) { return BF ? (u ? bf16_hi(w) : bf16_lo(w)) : __uint_as_float(w); };
  float s[JL] = {}, q[JL] = {};
  // (two j of a lane as one packed value; per j the order of the sums is that of the channels)
  float2 s2 = make_float2(0.f, 0.f), q2 = s2;
  const X* col = src + warp * 8 * chan;
  for (int g = warp; g < groups; g += LNT_WARPS, col += LNT_WARPS * 8 * chan) {
    uint32_t w[8];
    const X* p = col;
#pragma unroll
    for (int e = 0; e < 8; ++e, p += chan) w[e] = reinterpret_cast<const uint32_t*>(p)[lane];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      tile[(g * 8 + e) * 32 + lane] = w[e];
      if constexpr (BF)
        s2 = __fadd2_rn(s2, make_float2(bf16_lo(w[e]), bf16_hi(w[e])));
      else
        s[0] += __uint_as_float(w[e]);
    }
  }
  if constexpr (BF) {
    s[0] = s2.x;
    s[JL - 1] = s2.y;
  }
#pragma unroll
  for (int u = 0; u < JL; ++u) part[(warp * JL + u) * 32 + lane] = s[u];
  __syncthreads();
  const Channels chans(c_h);
#pragma unroll
  for (int u = 0; u < JL; ++u) {
    s[u] = 0.f;
#pragma unroll
    for (int w = 0; w < LNT_WARPS; ++w) s[u] += part[(w * JL + u) * 32 + lane];
    s[u] = chans.mean(s[u]);
  }
  const float2 minus_mean = make_float2(-s[0], -s[JL - 1]);
  for (int g = warp; g < groups; g += LNT_WARPS)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t w = tile[(g * 8 + e) * 32 + lane];  // (this thread's own words)
      if constexpr (BF) {
        const float2 d = __fadd2_rn(make_float2(bf16_lo(w), bf16_hi(w)), minus_mean);
        q2 = __ffma2_rn(d, d, q2);
      } else {
        const float d = __uint_as_float(w) - s[0];
        q[0] = fmaf(d, d, q[0]);
      }
    }
  if constexpr (BF) {
    q[0] = q2.x;
    q[JL - 1] = q2.y;
  }
  float* part_q = part + LNT_WARPS * JL * 32;
#pragma unroll
  for (int u = 0; u < JL; ++u) part_q[(warp * JL + u) * 32 + lane] = q[u];
  __syncthreads();
#pragma unroll
  for (int u = 0; u < JL; ++u) {
    q[u] = 0.f;
#pragma unroll
    for (int w = 0; w < LNT_WARPS; ++w) q[u] += part_q[(w * JL + u) * 32 + lane];
    q[u] = 1.0f / sqrtf(chans.mean(q[u]) + eps);
  }
  const float2 rstd = make_float2(q[0], q[JL - 1]);
  const X* scale = static_cast<const X*>(scale_);
  const X* bias = static_cast<const X*>(bias_);
  if constexpr (!BF && G > 0) {
    const int pitch = (groups + 7) & ~7;  // (as below)
    uint4* rows = reinterpret_cast<uint4*>(affine + (c_h + 63) / 64 * 64);
    for (int g = warp; g < groups; g += LNT_WARPS) {
      uint32_t w[3][4];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const int c = g * 8 + e;
        float v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          v[u] = (__uint_as_float(tile[(c + u) * 32 + lane]) - s[0]) * q[0] * static_cast<float>(scale[c + u]) +
                 static_cast<float>(bias[c + u]);
        split3x2(v[0], v[1], w[0][e / 2], w[1][e / 2], w[2][e / 2]);
      }
#pragma unroll
      for (int x = 0; x < 3; ++x)
        rows[(x * 32 + lane) * pitch + (g ^ (lane & 7))] = make_uint4(w[x][0], w[x][1], w[x][2], w[x][3]);
    }
    __syncthreads();
    const int count = min(JT, n - j0) * groups;
    for (int x = 0; x < 3; ++x) {
      uint4* dst = reinterpret_cast<uint4*>(tn + x * pairs * c_h + ((static_cast<long long>(b) * n + i) * n + j0) * c_h);
      for (int idx = threadIdx.x; idx < count; idx += LNT_WARPS * 32) {
        const int j = idx / groups, g = idx - j * groups;
        dst[idx] = rows[(x * 32 + j) * pitch + (g ^ (j & 7))];
      }
    }
    return;
  }
  if constexpr (BF && G > 0) {
    uint4 out[G][JL];
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int g = warp + k * LNT_WARPS;
      if (g >= groups) continue;
      uint32_t o[JL][4];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {  // two channels of two j, turned round
        uint32_t y[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const uint32_t w = tile[(g * 8 + e + u) * 32 + lane];
          const uint2 sb = affine[g * 8 + e + u];
          y[u] = affine_bf16x2(__fadd2_rn(make_float2(bf16_lo(w), bf16_hi(w)), minus_mean), rstd, sb.x, sb.y);
        }
        o[0][e / 2] = __byte_perm(y[0], y[1], 0x5410);
        o[JL - 1][e / 2] = __byte_perm(y[0], y[1], 0x7632);
      }
#pragma unroll
      for (int u = 0; u < JL; ++u) out[k][u] = make_uint4(o[u][0], o[u][1], o[u][2], o[u][3]);
    }
    __syncthreads();
    // rows of `pitch` 16-byte chunks, chunks swapped by the lane that writes them: no bank conflicts
    const int pitch = (groups + 7) & ~7;
    uint4* rows = reinterpret_cast<uint4*>(tile);
#pragma unroll
    for (int k = 0; k < G; ++k) {
      const int g = warp + k * LNT_WARPS;
      if (g >= groups) continue;
#pragma unroll
      for (int u = 0; u < JL; ++u) rows[(lane * JL + u) * pitch + (g ^ (lane & 7))] = out[k][u];
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(tn + ((static_cast<long long>(b) * n + i) * n + j0) * c_h);
    const int count = min(JT, n - j0) * groups;
    for (int idx = threadIdx.x; idx < count; idx += LNT_WARPS * 32) {
      const int j = idx / groups, g = idx - j * groups;
      dst[idx] = rows[j * pitch + (g ^ ((j / JL) & 7))];
    }
    return;
  }
  __nv_bfloat16* dst = tn + ((static_cast<long long>(b) * n + i) * n + j0 + lane * JL) * c_h;
  for (int g = warp; g < groups; g += LNT_WARPS) {
    float v[JL][8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int c = g * 8 + e;
      const uint32_t w = tile[c * 32 + lane];
      const float sc = static_cast<float>(scale[c]), bi = static_cast<float>(bias[c]);
#pragma unroll
      for (int u = 0; u < JL; ++u)
        v[u][e] = Rb<BF>::r(Rb<BF>::r(Rb<BF>::r((value(w, u) - s[u]) * q[u]) * sc) + bi);
    }
#pragma unroll
    for (int u = 0; u < JL; ++u)
      if (j0 + lane * JL + u < n) store_eight<BF ? 1 : 3>(dst + u * c_h + g * 8, pairs * c_h, v[u]);
  }
}

// The same in bf16, up to 64 * G channels: a lane's words stay in its registers from the load, all of
// them requested at once, to the result. (Through shared memory and in two batches of loads the 128
// channels of four 200-token templates took 36 us at 2.7 TB/s, and 25 so. With 384 channels it is the other
// way round, 27 us for 256 tokens and 29 in the registers of 16 warps.)
template <int G>
__global__ void __launch_bounds__(LNT_WARPS * 32, 4)
ln_channel_major_bf16_kernel(const __nv_bfloat16* __restrict__ t, int n, int ld, int c_h, const unsigned short* __restrict__ scale,
                             const unsigned short* __restrict__ bias, float eps, __nv_bfloat16* __restrict__ tn) {
  constexpr int JT = 64;
  extern __shared__ uint32_t tile[];  // the results, then partial sums, scale and bias (each twice in a word)
  float2* part = reinterpret_cast<float2*>(tile + (c_h + 63) / 64 * 64 * 32);
  uint2* affine = reinterpret_cast<uint2*>(part + 2 * LNT_WARPS * 32);
  pdl_wait();
  pdl_trigger();
  const int i = blockIdx.y, b = blockIdx.z, j0 = blockIdx.x * JT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, groups = c_h / 8;
  const long long chan = static_cast<long long>(n) * ld;
  const __nv_bfloat16* col = t + (static_cast<long long>(b) * c_h * n + i) * ld + j0 + warp * 8 * chan;
  uint32_t w[G][8];
#pragma unroll
  for (int k = 0; k < G; ++k, col += LNT_WARPS * 8 * chan) {
    const __nv_bfloat16* p = col;
#pragma unroll
    for (int e = 0; e < 8; ++e, p += chan)
      w[k][e] = warp + k * LNT_WARPS < groups ? reinterpret_cast<const uint32_t*>(p)[lane] : 0u;
  }
  for (int c = threadIdx.x; c < c_h; c += LNT_WARPS * 32) {
    const uint32_t sc = scale[c], bi = bias[c];
    affine[c] = make_uint2(sc | sc << 16, bi | bi << 16);
  }
  const Channels chans(c_h);
  float2 sum = make_float2(0.f, 0.f), var = sum;
#pragma unroll
  for (int k = 0; k < G; ++k)
#pragma unroll
    for (int e = 0; e < 8; ++e) sum = __fadd2_rn(sum, make_float2(bf16_lo(w[k][e]), bf16_hi(w[k][e])));
  part[warp * 32 + lane] = sum;
  __syncthreads();
  sum = make_float2(0.f, 0.f);
#pragma unroll
  for (int x = 0; x < LNT_WARPS; ++x) sum = __fadd2_rn(sum, part[x * 32 + lane]);
  const float2 minus_mean = make_float2(-chans.mean(sum.x), -chans.mean(sum.y));
#pragma unroll
  for (int k = 0; k < G; ++k)
    if (warp + k * LNT_WARPS < groups)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 d = __fadd2_rn(make_float2(bf16_lo(w[k][e]), bf16_hi(w[k][e])), minus_mean);
        var = __ffma2_rn(d, d, var);
      }
  float2* part_var = part + LNT_WARPS * 32;
  part_var[warp * 32 + lane] = var;
  __syncthreads();
  var = make_float2(0.f, 0.f);
#pragma unroll
  for (int x = 0; x < LNT_WARPS; ++x) var = __fadd2_rn(var, part_var[x * 32 + lane]);
  const float2 rstd = make_float2(1.0f / sqrtf(chans.mean(var.x) + eps), 1.0f / sqrtf(chans.mean(var.y) + eps));
  // rows of `pitch` 16-byte chunks, chunks swapped by the lane that writes them: no bank conflicts
  const int pitch = (groups + 7) & ~7;
  uint4* rows = reinterpret_cast<uint4*>(tile);
#pragma unroll
  for (int k = 0; k < G; ++k) {
    const int g = warp + k * LNT_WARPS;
    if (g >= groups) continue;
    uint32_t o[2][4];
#pragma unroll
    for (int e = 0; e < 8; e += 2) {  // two channels of two j, turned round
      uint32_t y[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint2 sb = affine[g * 8 + e + u];
        y[u] = affine_bf16x2(__fadd2_rn(make_float2(bf16_lo(w[k][e + u]), bf16_hi(w[k][e + u])), minus_mean), rstd, sb.x, sb.y);
      }
      o[0][e / 2] = __byte_perm(y[0], y[1], 0x5410);
      o[1][e / 2] = __byte_perm(y[0], y[1], 0x7632);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      rows[(lane * 2 + u) * pitch + (g ^ (lane & 7))] = make_uint4(o[u][0], o[u][1], o[u][2], o[u][3]);
  }
  __syncthreads();
  uint4* dst = reinterpret_cast<uint4*>(tn + ((static_cast<long long>(b) * n + i) * n + j0) * c_h);
  const int count = min(JT, n - j0) * groups;
  for (int idx = threadIdx.x; idx < count; idx += LNT_WARPS * 32) {
    const int j = idx / groups, g = idx - j * groups;
    dst[idx] = rows[j * pitch + (g ^ ((j / 2) & 7))];
  }
}

template <bool BF>
int launch_ln_channel_major(const void* t, int n, int batch, int ld, int c_h, const void* scale, const void* bias, float eps,
                            __nv_bfloat16* tn, cudaStream_t stream) {
  const dim3 grid((n + lnt_j<BF>() - 1) / lnt_j<BF>(), static_cast<unsigned>(n), static_cast<unsigned>(batch));
  auto go = [&](auto kernel, int staged = 0) {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), staged ? lnt_smem(384) + 384 * 192 : lnt_smem(1024));
    if (rc) return rc;
    return launch(kernel, grid, dim3(LNT_WARPS * 32), lnt_smem(round_up(c_h, 64)) + staged, stream, true, t, n, ld, c_h, scale, bias, eps,
                  static_cast<long long>(batch) * n * n, tn);
  };
  if constexpr (BF) {
    auto go_bf16 = [&](auto kernel) {
      const int smem = lnt_smem(round_up(c_h, 64)), rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), lnt_smem(128));
      if (rc) return rc;
      return launch(kernel, grid, dim3(LNT_WARPS * 32), smem, stream, true, static_cast<const __nv_bfloat16*>(t), n, ld, c_h,
                    static_cast<const unsigned short*>(scale), static_cast<const unsigned short*>(bias), eps, tn);
    };
    if (c_h <= 64) return go_bf16(ln_channel_major_bf16_kernel<1>);
    if (c_h <= 128) return go_bf16(ln_channel_major_bf16_kernel<2>);
    if (c_h <= 384) return go(ln_channel_major_kernel<BF, 6>);
  } else if (c_h <= 384) {
    return go(ln_channel_major_kernel<BF, 1>, round_up(c_h, 64) * 192);
  }
  return go(ln_channel_major_kernel<BF, 0>);
}

// ------------------------------------------------------------------- product policies
// Rows of pieces addressed as (batch, outer, inner): one box is `box` successive inner positions.
int map_rows(CUtensorMap* out, const void* base, int k, int n, long long s_inner, long long s_outer, int batch,
             int pieces, long long s_piece, int box) {
  const uint64_t un = n;
  const uint64_t dims[5] = {static_cast<uint64_t>(k), un, un, static_cast<uint64_t>(batch), static_cast<uint64_t>(pieces)};
  const uint64_t str[4] = {static_cast<uint64_t>(s_inner) * 2, static_cast<uint64_t>(s_outer) * 2,
                           un * un * static_cast<uint64_t>(k) * 2, static_cast<uint64_t>(s_piece) * 2};
  const uint32_t bx[5] = {GEMM_BK, static_cast<uint32_t>(box), 1, 1, 1};
  return make_tmap(out, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, bx, Swz::B128);
}

// A bf16 row's share of an epilogue warp, one row per thread: requested before the accumulators are
// waited for. Loaded after them it cost a gate tile two memory latencies, most of its time.
template <int COLS>
struct RowPrefetch {
  static_assert(COLS % 16 == 0, "whole sectors");
  uint4 row[COLS / 8];
  // `left` columns exist. `sectors`: rows start on 32-byte boundaries and have whole runs of 16 columns,
  // which then are one access: half an L2 sector at a time, what 128 rows of a tile cost the load/store
  // unit and L2 was most of a product's epilogue.
  __device__ __forceinline__ void load(const __nv_bfloat16* src, int left, bool sectors) {
    if (sectors) {
#pragma unroll
      for (int q = 0; q < COLS / 8; q += 2) {
        row[q] = row[q + 1] = make_uint4(0u, 0u, 0u, 0u);
        if (8 * q < left) load_sector(src + 8 * q, row[q], row[q + 1]);
      }
      return;
    }
#pragma unroll
    for (int q = 0; q < COLS / 8; ++q)
      row[q] = 8 * q < left ? reinterpret_cast<const uint4*>(src)[q] : make_uint4(0u, 0u, 0u, 0u);
  }
  // Eight neighbouring values rounded to bf16, with the prefetched residual added (one more rounding).
  __device__ __forceinline__ uint4 rounded(int q, bool residual, const float* v) const {
    uint4 u = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
    if (residual)
      u = make_uint4(bf16x2_add(row[q].x, u.x), bf16x2_add(row[q].y, u.y), bf16x2_add(row[q].z, u.z), bf16x2_add(row[q].w, u.w));
    return u;
  }
  // Sixteen of them, `left` of which exist.
  __device__ __forceinline__ void store(__nv_bfloat16* dst, int q, bool residual, const float* v, int left, bool sectors) const {
    const uint4 a = rounded(q, residual, v), b = rounded(q + 1, residual, v + 8);
    if (sectors) {
      store_sector(dst, a, b);
      return;
    }
    *reinterpret_cast<uint4*>(dst) = a;
    if (left > 8) reinterpret_cast<uint4*>(dst)[1] = b;
  }
};

// The same of a float32 row (256- and 150-token float32 stacks 860 -> 855 and 432 -> 426 us against loads behind the accumulators;
// 849 and 424 with no accumulator that K of 128 leaves unused).
template <int COLS>
struct RowPrefetchF {
  uint4 row[COLS / 4];
  __device__ __forceinline__ void load(const float* src, int left, bool sectors) {
#pragma unroll
    for (int q = 0; q < COLS / 4; q += 2) {
      row[q] = row[q + 1] = make_uint4(0u, 0u, 0u, 0u);
      if (4 * q >= left) continue;  // (a multiple of eight)
      if (sectors) {
        load_sector(src + 4 * q, row[q], row[q + 1]);
      } else {
        row[q] = reinterpret_cast<const uint4*>(src)[q];
        row[q + 1] = reinterpret_cast<const uint4*>(src)[q + 1];
      }
    }
  }
  __device__ __forceinline__ float at(int e) const {
    const uint4& w = row[e / 4];
    return __uint_as_float(e % 4 == 0 ? w.x : e % 4 == 1 ? w.y : e % 4 == 2 ? w.z : w.w);
  }
};

// Tile `tile` of rows walked `box` inner positions at a time.
struct RowTile {
  int b, o, t0;
  __device__ RowTile(uint32_t tile, const Divisor& n, const Divisor& tiles_t, int box) {
    const uint32_t bo = tiles_t.quotient(tile), bb = n.quotient(bo);
    t0 = static_cast<int>(tile - bo * tiles_t.d) * box;
    o = static_cast<int>(bo - bb * n.d);
    b = static_cast<int>(bb);
  }
};

// [a|b] = R(R(sigmoid(xn g)) * (xn p)) * mask, channel-major planes [piece][b * c_h + channel][o][ld].
// Transposed product (a TMEM lane is a channel of the 2 * c_h, segment 0 the values, 1 the
// gates), so that a thread stores runs of neighbouring pairs.
template <int PIECES, int NM, bool RES = false>
struct GluPolicy {
  static constexpr int BN = PIECES == 1 ? 128 : 64, PA = PIECES, PB = PIECES, NSEG = 2, NMAIN = NM;
  static constexpr bool TURNS = false;  // (in turn: 42 us instead of 40 for four 200-token templates)
  static constexpr bool A_MN = true, B_MN = false, M_FAST = true;
  static constexpr int EPI = PIECES == 1 && !RES ? 8 : 16, CTAS = PIECES == 1 && !RES ? 2 : 1;
  struct Params {
    int n, c_h, ld;
    Divisor by_n, tiles_t;
    long long piece;  // elements between pieces of a plane set
    const float* mask;
    long long ms_b, ms_o, ms_i;
    __nv_bfloat16 *a, *b;
  };
  static __device__ void load_a(const GemmMaps& maps, const Params&, int seg, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    gemm_load_mn(&maps.a[seg], dst, bar, 2, m_tile * GEMM_BM, k, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params& p, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    const RowTile r(n_tile, p.by_n, p.tiles_t, BN);
    tma_load_5d(dst, &maps.b[0], bar, k, r.t0, r.o, r.b, piece);
  }
  static constexpr bool BF = PIECES == 1;
  struct Pre {
    float mask[BN / (EPI / 4) / 16];  // of pair lane & 15 of each run of 16
  };
  static __device__ void prefetch(const Params& p, int, int n_tile, int, int col0, int, int lane, Pre& pre) {
    const RowTile rt(n_tile, p.by_n, p.tiles_t, BN);
#pragma unroll
    for (int i = 0; i < BN / (EPI / 4) / 16; ++i) {
      const int t = rt.t0 + col0 + 16 * i + (lane & 15);
      pre.mask[i] = p.mask && t < p.n ? p.mask[rt.b * p.ms_b + rt.o * p.ms_o + t * p.ms_i] : 1.0f;
    }
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<GluPolicy>& acc, int quarter,
                                  int col0, int, int lane, const Pre& pre) {
    const RowTile rt(n_tile, p.by_n, p.tiles_t, BN);
    const int c = m_tile * GEMM_BM + quarter * 32 + lane;
    const int chan = c < p.c_h ? c : c - p.c_h;
    __nv_bfloat16* dst = (c < p.c_h ? p.a : p.b) +
                         ((static_cast<long long>(rt.b) * p.c_h + chan) * p.n + rt.o) * p.ld + rt.t0;
#pragma unroll
    for (int i = 0; i < BN / (EPI / 4) / 16; ++i) {
      const int col = col0 + 16 * i;
      if (rt.t0 + col >= p.n) break;
      const float mk = pre.mask[i];
      float v[16], g[16];
      acc.load(0, col, v);
      acc.load(1, col, g);
      // (the pitch is a multiple of 64: the padding takes what lies past n)
      if constexpr (BF) {
        uint32_t u[8];
#pragma unroll
        for (int e = 0; e < 16; e += 2) u[e / 2] = bf16x2_mul(sigmoid_bf16x2(g[e], g[e + 1]), pack_bf16x2(v[e], v[e + 1]));
        if (!__all_sync(0xffffffffu, mk == 1.0f)) {  // (a factor of one changes nothing)
          const uint32_t mk2 = pack_bf16x2(mk, __shfl_down_sync(0xffffffffu, mk, 1));  // of two pairs, in the lane of the first
#pragma unroll
          for (int e = 0; e < 16; e += 2) u[e / 2] = bf16x2_mul(u[e / 2], __shfl_sync(0xffffffffu, mk2, e));
        }
        // a lane's 16 pairs are a whole sector of its channel
        if (c < 2 * p.c_h) store_sector(dst + col, make_uint4(u[0], u[1], u[2], u[3]), make_uint4(u[4], u[5], u[6], u[7]));
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = sigmoid_exact(g[e]) * v[e];
        if (!__all_sync(0xffffffffu, mk == 1.0f)) {
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] *= __shfl_sync(0xffffffffu, mk, e);
        }
        if (c < 2 * p.c_h) store_sixteen<PIECES>(dst + col, p.piece, v);
      }
    }
  }
};

// out = R(R(tn p_out) * R(sigmoid(R(xn g_out)))) (+ residual)
// Here and in the two products behind the attention core a tile of 128 bf16 columns has an SM with 16 epilogue warps to itself: as two
// CTAs of eight (in this product without a second pair of accumulators) 384-channel refiners of 64 / 100 / 150 tokens took 167 / 241 /
// 482 us, 159 / 232 / 466 so; 256 tokens the same.
template <int PIECES, int NM, int BN_>
struct OutGatePolicy {
  static constexpr int BN = BN_, PA = PIECES, PB = PIECES, NSEG = 2, NMAIN = NM;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = PIECES == 1 && BN <= 64 ? 8 : 16, CTAS = PIECES == 1 && BN <= 64 ? 2 : 1;
  static constexpr bool BF = PIECES == 1;
  // A float32 row beside three leading accumulators is more than the registers hold: asked for ahead of them, 68 bytes of spills and,
  // with or without a residual, 192 channels of 200 / 256 tokens 93 / 118 and 87 / 110 us, 92 / 119 and 76 / 96 behind them. Beside
  // one, 128 channels of 256 tokens 39.7 against 43.7, without a residual 36.1 both.
  static constexpr bool EARLY = BF || NM == 1;
  using O = typename std::conditional<BF, __nv_bfloat16, float>::type;
  struct Params {
    int n, c_z;
    Divisor by_n, tiles_j;
    const O* res;
    O* out;
    bool aligned, sectors;  // 16-byte and 32-byte accesses
  };
  using Pre = typename std::conditional<BF, RowPrefetch<BN / (EPI / 4)>, RowPrefetchF<BN / (EPI / 4)>>::type;
  static __device__ void prefetch(const Params& p, int m_tile, int n_tile, int quarter, int col0, int, int lane, Pre& pre) {
    if (!EARLY || !p.res || !p.aligned) return;
    const RowTile rt(m_tile, p.by_n, p.tiles_j, GEMM_BM);
    const int j = rt.t0 + quarter * 32 + lane, c0 = n_tile * BN + col0;
    pre.load(p.res + ((static_cast<long long>(rt.b) * p.n + rt.o) * p.n + j) * p.c_z + c0, j < p.n ? p.c_z - c0 : 0, p.sectors);
  }
  static __device__ void load_a(const GemmMaps& maps, const Params& p, int seg, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    const RowTile r(m_tile, p.by_n, p.tiles_j, GEMM_BM);
    tma_load_5d(dst, &maps.a[seg], bar, k, r.t0, r.o, r.b, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params&, int seg, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    gemm_load_mn(&maps.b[seg], dst, bar, BN / 64, n_tile * BN, k, piece);
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<OutGatePolicy>& acc, int quarter,
                                  int col0, int, int lane, const Pre& pre) {
    const RowTile rt(m_tile, p.by_n, p.tiles_j, GEMM_BM);
    const int j = rt.t0 + quarter * 32 + lane;
    const long long off = ((static_cast<long long>(rt.b) * p.n + rt.o) * p.n + j) * p.c_z;
#pragma unroll(BF ? 4 : 1)
    for (int i = 0; i < BN / (EPI / 4) / 16; ++i) {
      const int col = col0 + 16 * i, c0 = n_tile * BN + col;
      if (c0 >= p.c_z) break;
      float v[16], g[16];
      acc.load(0, col, v);
      acc.load(1, col, g);
      if (j >= p.n) continue;
#pragma unroll
      for (int e = 0; e < 16; e += 2) {
        if (BF) {
          const uint32_t u = bf16x2_mul(pack_bf16x2(v[e], v[e + 1]), sigmoid_bf16x2(g[e], g[e + 1]));
          v[e] = bf16_lo(u);
          v[e + 1] = bf16_hi(u);
        } else {
          v[e] *= sigmoid_exact(g[e]);
          v[e + 1] *= sigmoid_exact(g[e + 1]);
        }
      }
      if constexpr (BF) {
        if (p.aligned) {
          pre.store(p.out + off + c0, 2 * i, p.res != nullptr, v, p.c_z - c0, p.sectors);
          continue;
        }
      }
      const bool there = EARLY && !BF && p.res && p.aligned;  // the residual has been asked for
      if constexpr (!BF) {
        if (there)
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = pre.at(16 * i + e) + v[e];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (c0 + 8 * q < p.c_z)
          store_out<BF>(p.out + off + c0 + 8 * q, p.res && !there ? p.res + off + c0 + 8 * q : nullptr, v + 8 * q, p.aligned, p.sectors);
    }
  }
};

// q / sqrt(d), k: rows [piece][pair][hd]. v: transposed, [piece][(b, o)][hd][ld]. bias: [b][head][o][ld] in the trunk dtype. Column tiles walk
// the four weights in turn, in groups of 64 (so that narrow heads have tiles of 128 columns too).
template <int PIECES, int NM, int BN_, bool RES = false>
struct QkvbPolicy : NoPrefetch {
  static constexpr int BN = BN_, PA = PIECES, PB = PIECES, NSEG = 1, NMAIN = NM;
  static constexpr bool TURNS = true;  // tiles with the bias end in columns that do not exist: 28.0 -> 25.5 us
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = PIECES == 1 && !RES ? 8 : 16, CTAS = PIECES == 1 && !RES ? 2 : 1;
  static constexpr bool BF = PIECES == 1;
  struct Params {
    int n, hd, heads, groups_w, ld;  // groups_w: groups of 64 columns of a weight
    Divisor by_n;
    uint32_t pairs;
    float q_scale, q_scale_inv;
    long long row_piece, v_piece;  // elements between pieces of q / k and of v
    __nv_bfloat16 *q, *k, *vt;
    void* bias;
  };
  static __device__ int which(const Params& p, int group) {
    return (group >= p.groups_w) + (group >= 2 * p.groups_w) + (group >= 3 * p.groups_w);
  }
  static __device__ void load_a(const GemmMaps& maps, const Params& p, int, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    tma_load_3d(dst, &maps.a[0], bar, k, m_tile * GEMM_BM, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params& p, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
#pragma unroll
    for (int g = 0; g < BN / 64; ++g) {  // (a group behind the last one is columns that its map does not have: zeros)
      const int group = n_tile * (BN / 64) + g, w = which(p, group);
      gemm_load_mn(&maps.b[w], dst + g * 8192, bar, 1, (group - w * p.groups_w) * 64, k, piece);
    }
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<QkvbPolicy>& acc, int quarter,
                                  int col0, int col1, int lane, const Pre&) {
    const uint32_t pair = static_cast<uint32_t>(m_tile) * GEMM_BM + quarter * 32 + lane, n = p.n;
    const uint32_t bo = p.by_n.quotient(pair), t = pair - bo * n, b = p.by_n.quotient(bo), o = bo - b * n;
    // a warp's columns are those of one weight
    static_assert(64 % (BN / (EPI / 4)) == 0, "");
    const int group = n_tile * (BN / 64) + col0 / 64, w = which(p, group);
#pragma unroll 1
    for (int col = col0; col < col1; col += 16) {
      const int c0 = (group - w * p.groups_w) * 64 + col % 64;
      if (c0 >= (w == 3 ? p.heads : p.hd)) break;
      float v[16];
      acc.load(0, col, v);
      if (pair >= p.pairs) continue;
      if (w < 2) {
        __nv_bfloat16* dst = (w ? p.k : p.q) + static_cast<long long>(pair) * p.hd + c0;
        if (w == 0)
#pragma unroll
          // bf16: the product with the rounded reciprocal rounds like the quotient. The divisor is an odd
          // integer below 256 times a power of two and the dividend has 8 bits, so that the quotient is
          // representable or at least 1e-5 away from a rounding boundary.
          for (int e = 0; e < 16; ++e) v[e] = BF ? round_bf16(v[e]) * p.q_scale_inv : v[e] / p.q_scale;
        if (p.hd % 16 == 0) {
          store_sixteen<PIECES>(dst, p.row_piece, v);
          continue;
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if (c0 + 8 * q < p.hd) store_eight<PIECES>(dst + 8 * q, p.row_piece, v + 8 * q);
      } else if (w == 2) {
        __nv_bfloat16* dst = p.vt + (static_cast<long long>(bo) * p.hd + c0) * p.ld + t;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (c0 + e >= p.hd) break;
          if (BF) {
            dst[static_cast<long long>(e) * p.ld] = __float2bfloat16_rn(v[e]);
          } else {
            __nv_bfloat16* d = dst + static_cast<long long>(e) * p.ld;
            split3(v[e], d[0], d[p.v_piece], d[2 * p.v_piece]);
          }
        }
      } else {
        const long long at = (static_cast<long long>(b * p.heads + c0) * p.n + o) * p.ld + t;
        const long long head = static_cast<long long>(p.n) * p.ld;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          if (c0 + e >= p.heads) break;
          if (BF)
            static_cast<__nv_bfloat16*>(p.bias)[at + e * head] = __float2bfloat16_rn(v[e]);
          else
            static_cast<float*>(p.bias)[at + e * head] = v[e];
        }
      }
    }
  }
};

// y = R(o * R(sigmoid(R(xn Wg)))): bf16 in place over o, float32 o -> pieces
template <int PIECES, int NM, int BN_>
struct GatePolicy {
  static constexpr int BN = BN_, PA = PIECES, PB = PIECES, NSEG = 1, NMAIN = NM;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = PIECES == 1 && BN <= 64 ? 8 : 16, CTAS = PIECES == 1 && BN <= 64 ? 2 : 1;
  static constexpr bool BF = PIECES == 1;
  struct Params {
    long long pairs;
    int hd;
    const float* o;
    __nv_bfloat16* y;
  };
  using Pre = typename std::conditional<BF, RowPrefetch<BN / (EPI / 4)>, RowPrefetchF<BN / (EPI / 4)>>::type;
  static __device__ void prefetch(const Params& p, int m_tile, int n_tile, int quarter, int col0, int, int lane, Pre& pre) {
    const long long pair = static_cast<long long>(m_tile) * GEMM_BM + quarter * 32 + lane;
    const int c0 = n_tile * BN + col0;
    if constexpr (BF)
      pre.load(p.y + pair * p.hd + c0, pair < p.pairs ? p.hd - c0 : 0, p.hd % 16 == 0);
    else
      pre.load(p.o + pair * p.hd + c0, pair < p.pairs ? p.hd - c0 : 0, true);
  }
  static __device__ void load_a(const GemmMaps& maps, const Params&, int, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    tma_load_3d(dst, &maps.a[0], bar, k, m_tile * GEMM_BM, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params&, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    gemm_load_mn(&maps.b[0], dst, bar, BN / 64, n_tile * BN, k, piece);
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<GatePolicy>& acc, int quarter,
                                  int col0, int, int lane, const Pre& pre) {
    const long long pair = static_cast<long long>(m_tile) * GEMM_BM + quarter * 32 + lane;
#pragma unroll(BF ? 4 : 1)
    for (int i = 0; i < BN / (EPI / 4) / 16; ++i) {
      const int col = col0 + 16 * i, c0 = n_tile * BN + col;
      if (c0 >= p.hd) break;
      float g[16];
      acc.load(0, col, g);
      if (pair >= p.pairs) continue;
      const long long off = pair * p.hd + c0;
      if constexpr (BF) {
        uint4 w[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4 o = pre.row[2 * i + q];
          w[q].x = bf16x2_mul(o.x, sigmoid_bf16x2(g[8 * q + 0], g[8 * q + 1]));
          w[q].y = bf16x2_mul(o.y, sigmoid_bf16x2(g[8 * q + 2], g[8 * q + 3]));
          w[q].z = bf16x2_mul(o.z, sigmoid_bf16x2(g[8 * q + 4], g[8 * q + 5]));
          w[q].w = bf16x2_mul(o.w, sigmoid_bf16x2(g[8 * q + 6], g[8 * q + 7]));
        }
        if (p.hd % 16 == 0) {
          store_sector(p.y + off, w[0], w[1]);
        } else {
          *reinterpret_cast<uint4*>(p.y + off) = w[0];
          if (c0 + 8 < p.hd) reinterpret_cast<uint4*>(p.y + off)[1] = w[1];
        }
      } else {
        float v[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = pre.at(16 * i + e) * sigmoid_exact(g[e]);
        if (p.hd % 16 == 0) {
          store_sixteen<PIECES>(p.y + off, p.pairs * p.hd, v);
        } else {
#pragma unroll
          for (int q = 0; q < 2; ++q)
            if (c0 + 8 * q < p.hd) store_eight<PIECES>(p.y + off + 8 * q, p.pairs * p.hd, v + 8 * q);
        }
      }
    }
  }
};

// out[b][o * s_o + t * s_i] = R(y Wo) (+ residual): the ending node lands transposed back
template <int PIECES, int NM, int BN_>
struct ProjOutPolicy {
  static constexpr int BN = BN_, PA = PIECES, PB = PIECES, NSEG = 1, NMAIN = NM;
  static constexpr bool A_MN = false, B_MN = true, M_FAST = false;
  static constexpr int EPI = PIECES == 1 && BN <= 64 ? 8 : 16, CTAS = PIECES == 1 && BN <= 64 ? 2 : 1;
  static constexpr bool BF = PIECES == 1;
  using O = typename std::conditional<BF, __nv_bfloat16, float>::type;
  struct Params {
    long long pairs;
    int c_z;
    Divisor by_n;
    long long s_b, s_o, s_i;
    const O* res;
    O* out;
    bool aligned, sectors;  // 16-byte and 32-byte accesses
  };
  using Pre = typename std::conditional<BF, RowPrefetch<BN / (EPI / 4)>, RowPrefetchF<BN / (EPI / 4)>>::type;
  static __device__ long long offset(const Params& p, uint32_t pair) {
    const uint32_t n = p.by_n.d, bo = p.by_n.quotient(pair), t = pair - bo * n, b = p.by_n.quotient(bo), o = bo - b * n;
    return b * p.s_b + o * p.s_o + t * p.s_i;
  }
  static __device__ void prefetch(const Params& p, int m_tile, int n_tile, int quarter, int col0, int, int lane, Pre& pre) {
    if (!p.res || !p.aligned) return;
    const uint32_t pair = static_cast<uint32_t>(m_tile) * GEMM_BM + quarter * 32 + lane;
    const int c0 = n_tile * BN + col0;
    pre.load(p.res + offset(p, pair) + c0, pair < p.pairs ? p.c_z - c0 : 0, p.sectors);
  }
  static __device__ void load_a(const GemmMaps& maps, const Params&, int, int k, int m_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    tma_load_3d(dst, &maps.a[0], bar, k, m_tile * GEMM_BM, piece);
  }
  static __device__ void load_b(const GemmMaps& maps, const Params&, int, int k, int n_tile, int piece, uint8_t* dst,
                                uint64_t* bar) {
    gemm_load_mn(&maps.b[0], dst, bar, BN / 64, n_tile * BN, k, piece);
  }
  static __device__ void epilogue(const Params& p, int m_tile, int n_tile, int, const Accum<ProjOutPolicy>& acc, int quarter,
                                  int col0, int, int lane, const Pre& pre) {
    const uint32_t pair = static_cast<uint32_t>(m_tile) * GEMM_BM + quarter * 32 + lane;
    const long long off = offset(p, pair);
#pragma unroll(BF ? 4 : 1)
    for (int i = 0; i < BN / (EPI / 4) / 16; ++i) {
      const int col = col0 + 16 * i, c0 = n_tile * BN + col;
      if (c0 >= p.c_z) break;
      float v[16];
      acc.load(0, col, v);
      if (pair >= p.pairs) continue;
      if constexpr (BF) {
        if (p.aligned) {
          pre.store(p.out + off + c0, 2 * i, p.res != nullptr, v, p.c_z - c0, p.sectors);
          continue;
        }
      }
      const bool there = !BF && p.res && p.aligned;  // the residual has been asked for
      if constexpr (!BF) {
        if (there)
#pragma unroll
          for (int e = 0; e < 16; ++e) v[e] = pre.at(16 * i + e) + v[e];
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (c0 + 8 * q < p.c_z)
          store_out<BF>(p.out + off + c0 + 8 * q, p.res && !there ? p.res + off + c0 + 8 * q : nullptr, v + 8 * q, p.aligned, p.sectors);
    }
  }
};

int ksteps(int k) { return (k + GEMM_BK - 1) / GEMM_BK; }

// The product with both operands streamed, or with one kept (`keep`, where its k steps fit beside
// three stages of the other and there are several tiles to use it for).
template <class Streamed, class Resident>
int launch_either(const GemmMaps& maps, const GemmShape& g, const typename Streamed::Params& ep, bool keep,
                  cudaStream_t stream) {
  const int fast = Streamed::M_FAST ? g.m_tiles : g.n_tiles;
  if (keep && fast >= 2 && gemm_res_stages<Resident>(g.kb[0]) > 0) {
    typename Resident::Params r;
    static_assert(sizeof(r) == sizeof(ep), "the same arguments");
    memcpy(&r, &ep, sizeof(r));
    return launch_piece_gemm_resident<Resident>(maps, g, r, stream, true);
  }
  return launch_piece_gemm<Streamed>(maps, g, ep, stream, true);
}

// ------------------------------------------------------------------------- workspaces
struct Offsets {
  size_t off = 0;
  size_t take(size_t bytes) {
    off = (off + 1023) / 1024 * 1024;
    const size_t r = off;
    off += bytes;
    return r;
  }
  size_t total() const { return (off + 1023) / 1024 * 1024; }
};

struct TrimulPlan {
  size_t xn, ap, bp, t, tn, w[4], total;
};

TrimulPlan trimul_plan(int n, int batch, int c_z, int c_h, bool f32) {
  TrimulPlan pl;
  Offsets w;
  const size_t pairs = static_cast<size_t>(batch) * n * n, ld = round_up(n, 64), pieces = f32 ? 3 : 1;
  const size_t planes = static_cast<size_t>(batch) * c_h * n * ld;
  pl.xn = w.take(pieces * pairs * c_z * 2);
  pl.ap = w.take(pieces * planes * 2);
  pl.bp = w.take(pieces * planes * 2);
  pl.t = w.take(planes * (f32 ? 4 : 2));
  pl.tn = w.take(pieces * pairs * c_h * 2);
  pl.w[0] = w.take(pieces * c_z * 2 * c_h * 2);
  pl.w[1] = w.take(pieces * c_z * 2 * c_h * 2);
  pl.w[2] = w.take(pieces * c_h * c_z * 2);
  pl.w[3] = w.take(pieces * c_z * c_z * 2);
  pl.total = w.total();
  return pl;
}

struct TriattPlan {
  size_t xn, q, k, vt, bias, mb, o, y, w[6], total;
};

TriattPlan triatt_plan(int n, int batch, int c_z, int heads, int head_dim, bool f32) {
  TriattPlan pl;
  Offsets w;
  const size_t pairs = static_cast<size_t>(batch) * n * n, hd = static_cast<size_t>(heads) * head_dim;
  const size_t ld = round_up(n, 64), pieces = f32 ? 3 : 1, rows = static_cast<size_t>(batch) * n;
  pl.xn = w.take(pieces * pairs * c_z * 2);
  pl.q = w.take(pieces * pairs * hd * 2);
  pl.k = w.take(pieces * pairs * hd * 2);
  pl.vt = w.take(pieces * rows * hd * ld * 2);
  pl.bias = w.take(rows * heads * ld * (f32 ? 4 : 2));
  pl.mb = w.take(rows * ld * 4);
  pl.o = w.take(pairs * hd * (f32 ? 4 : 2));
  pl.y = f32 ? pl.q : pl.o;  // the gated output: over the queries, which the core has read, or in place
  for (int i = 0; i < 6; ++i) pl.w[i] = w.take(pieces * c_z * (i == 3 ? static_cast<size_t>(round_up(heads, 8)) : hd) * 2);
  pl.total = w.total();
  return pl;
}

// Batch items one pass can take with the workspace the caller gave: pair indices are 32-bit inside
// the kernels, and a grid's third dimension, which the layer norms count the items in, ends at 65535.
template <class F>
int items_per_pass(int batch, int n, size_t bytes, F total_of) {
  const long long by_pairs = 4000000000ll / (static_cast<long long>(n) * n);
  int low = 1, high = batch < 65535 ? batch : 65535;
  high = by_pairs < high ? static_cast<int>(by_pairs) : high;
  while (low < high) {  // the scratch grows with the items
    const int mid = high - (high - low) / 2;
    if (total_of(mid) <= bytes)
      low = mid;
    else
      high = mid - 1;
  }
  return low;
}

// Weights of one op: read in place where TMA can, else listed for one weight_kernel launch.
struct WeightStage {
  bool f32;
  WeightJobs jobs = {};
  int count = 0;
  int add(CUtensorMap* map, const void* w, int k, int n, uint8_t* scratch) {
    const int ld = round_up(n, 8);
    if (!f32 && n % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0) return gemm_map_mnmajor(map, w, k, n, n);
    jobs.job[count++] = {w, reinterpret_cast<__nv_bfloat16*>(scratch), k, n, ld};
    return gemm_map_mnmajor(map, scratch, k, n, ld, f32 ? 3 : 1);
  }
  int run(cudaStream_t stream) {
    if (!count) return B200TRI_OK;
    const dim3 grid(64, static_cast<unsigned>(count));
    return f32 ? launch(weight_kernel<false>, grid, dim3(256), 0, stream, true, jobs)
               : launch(weight_kernel<true>, grid, dim3(256), 0, stream, true, jobs);
  }
};

bool aligned32(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 31) == 0;
}
bool aligned16(const void* a, const void* b) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
}

template <bool BF>
int trimul_generic(const b200tri_trimul_args* a, int c_z, int c_h, cudaStream_t stream) {
  using O = typename std::conditional<BF, __nv_bfloat16, float>::type;
  constexpr int P = BF ? 1 : 3;
  const int n = a->n, batch = a->batch > 0 ? a->batch : 1;
  const int group = items_per_pass(batch, n, a->workspace_bytes, [&](int g) { return trimul_plan(n, g, c_z, c_h, !BF).total; });
  const TrimulPlan pl = trimul_plan(n, group, c_z, c_h, !BF);
  uint8_t* ws = static_cast<uint8_t*>(a->workspace);
  auto at = [&](size_t off) { return reinterpret_cast<__nv_bfloat16*>(ws + off); };
  GemmMaps glu = {}, fin = {};
  WeightStage weights{!BF};
  int rc;
  if ((rc = weights.add(&glu.a[0], a->p_in, c_z, 2 * c_h, ws + pl.w[0]))) return rc;
  if ((rc = weights.add(&glu.a[1], a->g_in, c_z, 2 * c_h, ws + pl.w[1]))) return rc;
  if ((rc = weights.add(&fin.b[0], a->p_out, c_h, c_z, ws + pl.w[2]))) return rc;
  if ((rc = weights.add(&fin.b[1], a->g_out, c_z, c_z, ws + pl.w[3]))) return rc;
  if ((rc = weights.run(stream))) return rc;
  const int ld = round_up(n, 64);
  const long long nn = static_cast<long long>(n) * n;
  for (int b0 = 0; b0 < batch; b0 += group) {
    const int nb = batch - b0 < group ? batch - b0 : group;
    const long long pairs = nb * nn, plane = static_cast<long long>(n) * ld, piece = nb * c_h * plane;
    const O* res = a->residual ? static_cast<const O*>(a->residual) + b0 * nn * c_z : nullptr;
    O* out = static_cast<O*>(a->out) + b0 * nn * c_z;
    const float* mask = a->mask ? a->mask + b0 * nn : nullptr;
    // projection frame (o, t): the outgoing update reads x[o][t], the incoming one x[t][o], so
    // both contract over t (triangle.py:231, :239)
    LnArgs ln = {};
    ln.x = static_cast<const O*>(a->x) + b0 * nn * c_z;
    ln.xs_b = nn * c_z;
    ln.xs_o = a->incoming ? c_z : static_cast<long long>(n) * c_z;
    ln.xs_i = a->incoming ? static_cast<long long>(n) * c_z : c_z;
    ln.batch = nb;
    ln.n = n;
    ln.c = c_z;
    ln.scale = a->norm_in_scale;
    ln.bias = a->norm_in_bias;
    ln.eps = a->eps;
    ln.xn = at(pl.xn);
    if ((rc = launch_ln_gather<BF>(ln, stream, true))) return rc;
    {
      constexpr int BN = GluPolicy<P, 1>::BN;
      if ((rc = map_rows(&glu.b[0], at(pl.xn), c_z, n, c_z, static_cast<long long>(n) * c_z, nb, P, pairs * c_z, BN))) return rc;
      const int tiles_t = (n + BN - 1) / BN;
      const GemmShape g = {(2 * c_h + GEMM_BM - 1) / GEMM_BM, nb * n * tiles_t, 1, {ksteps(c_z), ksteps(c_z)}, nullptr};
      auto go = [&](auto policy, auto kept) {
        using Pol = decltype(policy);
        return launch_either<Pol, decltype(kept)>(glu, g, {n, c_h, ld, Divisor(n), Divisor(tiles_t), piece, mask, nn, a->incoming ? 1ll : n,
                                               a->incoming ? n : 1ll, at(pl.ap), at(pl.bp)}, true, stream);
      };
      if constexpr (BF)
        rc = go(GluPolicy<1, 1>{}, GluPolicy<1, 1, true>{});
      else  // (a longer K wants its leading term in more accumulators than double buffering leaves room for)
        rc = c_z <= 128 ? go(GluPolicy<3, 1>{}, GluPolicy<3, 1, true>{}) : go(GluPolicy<3, 3>{}, GluPolicy<3, 3, true>{});
      if (rc) return rc;
    }
    {
      b200tri_trimul_contract_args ca = {};
      ca.n_i = ca.n_j = ca.n_k = n;
      ca.n_src = 1;
      ca.a = at(pl.ap);
      ca.b = at(pl.bp);
      ca.a_ld = ca.b_ld = ca.out_ld = ld;
      ca.a_chan_stride = ca.b_chan_stride = ca.out_chan_stride = plane;
      ca.a_src_stride = ca.b_src_stride = piece;
      if (BF)
        ca.out_bf16 = ws + pl.t;
      else
        ca.out_f32 = reinterpret_cast<float*>(ws + pl.t);
      const ContractTerms terms = BF ? ContractTerms{} : ContractTerms{6, {2, 0, 1, 1, 0, 0}, {0, 2, 1, 0, 1, 0}};
      if ((rc = contract_launch(&ca, nb * c_h, terms, true, stream))) return rc;
    }
    if ((rc = launch_ln_channel_major<BF>(ws + pl.t, n, nb, ld, c_h, a->norm_out_scale, a->norm_out_bias, a->eps, at(pl.tn),
                                          stream)))
      return rc;
    {
      // the gate's rows live in the projection frame: transposed for the incoming update
      const long long r1 = a->incoming ? static_cast<long long>(n) * c_z : c_z, r2 = a->incoming ? c_z : static_cast<long long>(n) * c_z;
      if ((rc = map_rows(&fin.a[0], at(pl.tn), c_h, n, c_h, static_cast<long long>(n) * c_h, nb, P, pairs * c_h, GEMM_BM))) return rc;
      if ((rc = map_rows(&fin.a[1], at(pl.xn), c_z, n, r1, r2, nb, P, pairs * c_z, GEMM_BM))) return rc;
      const int tiles_j = (n + GEMM_BM - 1) / GEMM_BM;
      auto go = [&](auto policy) {
        using Pol = decltype(policy);
        const GemmShape g = {nb * n * tiles_j, (c_z + Pol::BN - 1) / Pol::BN, 1, {ksteps(c_h), ksteps(c_z)}, nullptr};
        return launch_piece_gemm<Pol>(fin, g, {n, c_z, Divisor(n), Divisor(tiles_j), res, out, aligned16(out, res), (!BF || c_z % 16 == 0) && aligned32(out, res)}, stream, true);
      };
      if constexpr (BF)
        rc = c_z <= 64 ? go(OutGatePolicy<1, 1, 64>{}) : go(OutGatePolicy<1, 1, 128>{});
      else
        rc = c_z <= 128 && c_h <= 128 ? go(OutGatePolicy<3, 1, 64>{}) : go(OutGatePolicy<3, 3, 64>{});
      if (rc) return rc;
    }
  }
  return B200TRI_OK;
}

template <bool BF>
int triatt_generic(const b200tri_triatt_args* a, int c_z, cudaStream_t stream) {
  using O = typename std::conditional<BF, __nv_bfloat16, float>::type;
  constexpr int P = BF ? 1 : 3;
  const int n = a->n, heads = a->heads, head_dim = a->head_dim, hd = heads * head_dim, batch = a->batch > 0 ? a->batch : 1;
  const int group =
      items_per_pass(batch, n, a->workspace_bytes, [&](int g) { return triatt_plan(n, g, c_z, heads, head_dim, !BF).total; });
  const TriattPlan pl = triatt_plan(n, group, c_z, heads, head_dim, !BF);
  uint8_t* ws = static_cast<uint8_t*>(a->workspace);
  auto at = [&](size_t off) { return reinterpret_cast<__nv_bfloat16*>(ws + off); };
  GemmMaps proj = {}, gate = {}, outp = {};
  WeightStage weights{!BF};
  int rc;
  if ((rc = weights.add(&proj.b[0], a->w_q, c_z, hd, ws + pl.w[0]))) return rc;
  if ((rc = weights.add(&proj.b[1], a->w_k, c_z, hd, ws + pl.w[1]))) return rc;
  if ((rc = weights.add(&proj.b[2], a->w_v, c_z, hd, ws + pl.w[2]))) return rc;
  if ((rc = weights.add(&proj.b[3], a->w_bias, c_z, heads, ws + pl.w[3]))) return rc;
  if ((rc = weights.add(&gate.b[0], a->w_g, c_z, hd, ws + pl.w[4]))) return rc;
  if ((rc = weights.add(&outp.b[0], a->w_o, hd, c_z, ws + pl.w[5]))) return rc;
  if ((rc = weights.run(stream))) return rc;
  const int ld = round_up(n, 64);
  const long long nn = static_cast<long long>(n) * n;
  // attention frame (o = row, t = position inside the row): the ending node is the starting
  // node on the transposed pair tensor and mask (triangle_attention.py:128-130, :160-161)
  const long long s_o = a->starting ? static_cast<long long>(n) * c_z : c_z;
  const long long s_i = a->starting ? c_z : static_cast<long long>(n) * c_z;
  for (int b0 = 0; b0 < batch; b0 += group) {
    const int nb = batch - b0 < group ? batch - b0 : group;
    const long long pairs = nb * nn;
    const O* res = a->residual ? static_cast<const O*>(a->residual) + b0 * nn * c_z : nullptr;
    O* out = static_cast<O*>(a->out) + b0 * nn * c_z;
    float* mb = reinterpret_cast<float*>(ws + pl.mb);
    LnArgs ln = {};
    ln.x = static_cast<const O*>(a->x) + b0 * nn * c_z;
    ln.xs_b = nn * c_z;
    ln.xs_o = s_o;
    ln.xs_i = s_i;
    ln.batch = nb;
    ln.n = n;
    ln.c = c_z;
    ln.scale = a->norm_scale;
    ln.bias = a->norm_bias;
    ln.eps = a->eps;
    ln.xn = at(pl.xn);
    ln.mb = mb;
    ln.mask = a->mask ? a->mask + b0 * nn : nullptr;
    ln.ms_b = nn;
    ln.ms_o = a->starting ? n : 1;
    ln.ms_i = a->starting ? 1 : n;
    ln.inf = a->inf;
    ln.mb_ld = ld;
    if ((rc = launch_ln_gather<BF>(ln, stream, true))) return rc;
    const float root = sqrtf(static_cast<float>(head_dim));
    const int m_tiles = static_cast<int>((pairs + GEMM_BM - 1) / GEMM_BM);
    {
      if ((rc = gemm_map_kmajor(&proj.a[0], at(pl.xn), P, pairs, c_z, c_z, GEMM_BM))) return rc;
      auto go = [&](auto policy, auto kept) {
        using Pol = decltype(policy);
        const int groups_w = (hd + 63) / 64, groups = 3 * groups_w + (heads + 63) / 64;
        const GemmShape g = {m_tiles, (groups + Pol::BN / 64 - 1) / (Pol::BN / 64), 1, {ksteps(c_z), 0}, nullptr};
        const float q_scale = BF ? __bfloat162float(__float2bfloat16_rn(root)) : root;
        // Keeping the rows pays up to two k steps, and in bf16 with more where there are tiles enough for long runs: streamed,
        // 128 x 128 tiles take 64 bytes a clock and SM, all that L2 gives. Kept / streamed, us: refiner stacks (384 channels, 12 x 32
        // heads) of 300 / 256 / 200 / 150 / 100 tokens 1683 / 1697, 1053 / 1068, 731 / 732, 472 / 460, 243 / 230 (704 / 512 /
        // 313 / 176 / 79 tiles of rows); attention of as many channels as heads x 32, 192 / 256 / 320 / 384, at 256 tokens 147 / 154, 187 / 189,
        // 221 / 221, 281 / 295, the last three at 384 tokens 490 / 508, 610 / 625, 756 / 774; 4 heads x 16 at 256 tokens 109.8 / 110.1,
        // 114.3 / 114.9, 130.1 / 131.1, 140.2 / 141.5 (512 channels 176.6 / 177.4, left streaming); float32 attention of 128 channels, four
        // 200-token templates, 455 / 491, of 192 333 / 313.
        const bool keep = ksteps(c_z) <= 2 || (BF && ksteps(c_z) <= 6 && m_tiles >= 3 * sm_count());
        const typename Pol::Params params = {n, hd, heads, groups_w, ld, Divisor(n), static_cast<uint32_t>(pairs), q_scale, 1.0f / q_scale, pairs * hd,
                                             static_cast<long long>(nb) * n * hd * ld, at(pl.q), at(pl.k), at(pl.vt), ws + pl.bias};
        if constexpr (std::is_same<Pol, decltype(kept)>::value)
          return launch_piece_gemm<Pol>(proj, g, params, stream, true);
        else
          return launch_either<Pol, decltype(kept)>(proj, g, params, keep, stream);
      };
      // Narrow heads with little more than a tile of rows an SM: 64 columns, streamed, are four tiles to share among the SMs instead of two
      // (us with them and with 128 columns, 4 heads x 16, tokens: 64 channels of 64 / 100 / 150 4.3 / 5.7 / 9.0 and 5.2 / 6.3 / 10.1, 256
      // 5.4 / 8.4 / 15.0 and 6.3 / 9.5 / 16.0, 512 6.7 / 12.4 / 19.5 and 8.0 / 13.3 / 21.0; at 200 tokens, 313 tiles of rows, 64 / 192 / 256 /
      // 384 channels 15.9 / 21.0 / 23.9 / 31.3 and 14.2 / 21.6 / 23.8 / 29.5, at 256 19.9 / 30.4 / 36.4 / 41.3 and 15.6 / 28.5 / 32.6 / 36.5).
      if constexpr (BF)
        rc = hd <= 64 && 4ll * m_tiles <= 5ll * sm_count() ? go(QkvbPolicy<1, 1, 64>{}, QkvbPolicy<1, 1, 64>{})
                                                           : go(QkvbPolicy<1, 1, 128>{}, QkvbPolicy<1, 1, 128, true>{});
      else
        rc = ksteps(c_z) <= 2 ? go(QkvbPolicy<3, 2, 64>{}, QkvbPolicy<3, 2, 64, true>{}) : go(QkvbPolicy<3, 3, 64>{}, QkvbPolicy<3, 3, 64, true>{});
      if (rc) return rc;
    }
    {
      AttSplitArgs s = {};
      s.bf16 = BF;
      s.batch = nb;
      s.n_i = s.n = n;
      s.heads = heads;
      s.head_dim = head_dim;
      s.q = at(pl.q);
      s.k = at(pl.k);
      s.vt = at(pl.vt);
      s.v_ld = s.bias_ld = s.mask_ld = ld;
      s.bias = ws + pl.bias;
      s.mask_bias = mb;
      s.scale = 1.0f;
      s.o = ws + pl.o;
      s.pdl = true;
      if ((rc = launch_att_split(s, stream))) return rc;
    }
    {
      if ((rc = gemm_map_kmajor(&gate.a[0], at(pl.xn), P, pairs, c_z, c_z, GEMM_BM))) return rc;
      auto go = [&](auto policy) {
        using Pol = decltype(policy);
        const GemmShape g = {m_tiles, (hd + Pol::BN - 1) / Pol::BN, 1, {ksteps(c_z), 0}, nullptr};
        return launch_piece_gemm<Pol>(gate, g, {pairs, hd, reinterpret_cast<const float*>(ws + pl.o), at(pl.y)}, stream, true);
      };
      if constexpr (BF)
        rc = hd <= 64 ? go(GatePolicy<1, 1, 64>{})
                     : go(GatePolicy<1, 1, 128>{});
      else
        rc = ksteps(c_z) <= 2 ? go(GatePolicy<3, 2, 64>{}) : go(GatePolicy<3, 3, 64>{});
      if (rc) return rc;
    }
    {
      if ((rc = gemm_map_kmajor(&outp.a[0], at(pl.y), P, pairs, hd, hd, GEMM_BM))) return rc;
      auto go = [&](auto policy) {
        using Pol = decltype(policy);
        const GemmShape g = {m_tiles, (c_z + Pol::BN - 1) / Pol::BN, 1, {ksteps(hd), 0}, nullptr};
        return launch_piece_gemm<Pol>(outp, g, {pairs, c_z, Divisor(n), nn * c_z, s_o, s_i, res, out, aligned16(out, res), (!BF || c_z % 16 == 0) && aligned32(out, res)}, stream, true);
      };
      if constexpr (BF)
        rc = c_z <= 64 ? go(ProjOutPolicy<1, 1, 64>{})
                      : go(ProjOutPolicy<1, 1, 128>{});
      else
        rc = ksteps(hd) <= 2 ? go(ProjOutPolicy<3, 2, 64>{}) : go(ProjOutPolicy<3, 3, 64>{});
      if (rc) return rc;
    }
  }
  return B200TRI_OK;
}

}  // namespace

size_t trimul_workspace_bytes_generic(int32_t n, int32_t c_z, int32_t c_h, int32_t dtype) {
  if (n <= 0 || c_z <= 0 || c_h <= 0) return 0;
  return trimul_plan(n, 1, c_z, c_h, dtype == B200TRI_DTYPE_F32).total;
}

size_t triatt_workspace_bytes_generic(int32_t n, int32_t c_z, int32_t heads, int32_t head_dim, int32_t dtype) {
  if (n <= 0 || c_z <= 0 || heads <= 0 || head_dim <= 0) return 0;
  return triatt_plan(n, 1, c_z, heads, head_dim, dtype == B200TRI_DTYPE_F32).total;
}

int trimul_forward_generic(const b200tri_trimul_args* a, int c_z, int c_h, cudaStream_t stream) {
  B200_REQUIRE(a->n <= 65535, B200TRI_ERR_UNSUPPORTED, "trimul (general shapes): n up to 65535");
  return a->dtype == B200TRI_DTYPE_F32 ? trimul_generic<false>(a, c_z, c_h, stream)
                                       : trimul_generic<true>(a, c_z, c_h, stream);
}

int triatt_forward_generic(const b200tri_triatt_args* a, int c_z, cudaStream_t stream) {
  B200_REQUIRE(a->n <= 65535, B200TRI_ERR_UNSUPPORTED, "triatt (general shapes): n up to 65535");
  B200_REQUIRE(a->head_dim == 8 || a->head_dim == 16 || a->head_dim == 24 || a->head_dim == 32 || a->head_dim == 48 ||
                   a->head_dim == 64,
               B200TRI_ERR_UNSUPPORTED, "triatt: head widths 8, 16, 24, 32, 48 and 64 are built (got %d)", a->head_dim);
  return a->dtype == B200TRI_DTYPE_F32 ? triatt_generic<false>(a, c_z, stream) : triatt_generic<true>(a, c_z, stream);
}

}  // namespace b200
