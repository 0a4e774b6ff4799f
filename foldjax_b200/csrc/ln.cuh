// Layer norm of 128-channel pairs held in a K-major, 128-byte-swizzled operand tile (two 16 KiB
// slabs of 64 channels; row = pair). Statistics in fp32 as the reference takes them (mean, then mean
// of squared deviations, rsqrt(var + eps); src/foldjax/models/boltz2/models/primitives/
// _common.py:15-26), the normalised value rounded to bf16 before the affine step like the
// reference, the result written back in place: the tile TMA delivered becomes the tensor-core
// operand without a second buffer. The fp32 arithmetic runs two channels an instruction.
#pragma once
#include "tc.cuh"

namespace b200 {

constexpr int SLAB_BYTES = 128 * 128;  // 128 rows x 64 bf16

// Channel pair `i` of a bf16 layer-norm parameter, packed (any alignment).
__device__ __forceinline__ uint32_t ln_param_pair(const void* p, int i) {
  const unsigned short* h = static_cast<const unsigned short*>(p) + 2 * i;
  return static_cast<uint32_t>(h[0]) | (static_cast<uint32_t>(h[1]) << 16);
}
// The same, requested by one thread of the layer norm's warps as soon as it runs and put together when they have got
// to their role, beside the load of the first tile: waited for ahead of the block's first barrier it holds up
// everything else a launch begins with. (Not in the attention's projection and output stages, which it cost
// registers: 24 blocks of 200 tokens 5722 us without, 5748 with the former, 178 us against 166 a launch of the latter.)
struct LnParam {
  uint32_t lo, hi;
  __device__ __forceinline__ void request(const void* p, int i) {
    const unsigned short* h = static_cast<const unsigned short*>(p) + 2 * i;
    lo = h[0];
    hi = h[1];
  }
  __device__ __forceinline__ uint32_t word() {
    asm volatile("" : "+r"(lo), "+r"(hi));  // (not put together earlier)
    return lo | hi << 16;
  }
};

// The operations below and their order are part of the result: a statistic that differs in its last
// bit flips some roundings to bf16 later on, and a stack of blocks amplifies those. Where two
// operations of the same kind are independent they share an instruction, and a bf16 value is added by a mixed-precision
// fma instead of being unpacked for it (multiplication of 1003 tokens 737 -> 725 us, block of 203 278 -> 276, the same bits).

// normed.astype(bf16) * scale + bias, each step rounded to bf16
__device__ __forceinline__ uint32_t ln_affine(uint32_t w, float2 minus_mean, float2 rstd, uint32_t gamma, uint32_t beta) {
  const float2 n = __fmul2_rn(add_bf16x2(minus_mean, w), rstd);
  return bf16x2_add(bf16x2_mul(pack_bf16x2(n.x, n.y), gamma), beta);
}
// One step of each statistic in one accumulator: a word's two channels are added to each other
// first; their squared deviations one after the other.
__device__ __forceinline__ float ln_add4(float sum, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
  return (((sum + sum_bf16x2(w0)) + sum_bf16x2(w1)) + sum_bf16x2(w2)) + sum_bf16x2(w3);
}
__device__ __forceinline__ float ln_square(float sq, uint32_t w, float2 minus_mean) {
  const float2 d = add_bf16x2(minus_mean, w);
  return fmaf(d.y, d.y, fmaf(d.x, d.x, sq));
}

// One thread per row, the row's 64 packed words in registers. gamma2 / beta2: scale and bias as
// 64 packed bf16 pairs in shared memory, 16-byte aligned (every thread reads the same address, a
// broadcast).
__device__ __forceinline__ void ln_row_words(uint4 (&v)[16], const uint32_t* gamma2, const uint32_t* beta2, float eps) {
  float sum = 0.f, sq = 0.f;
#pragma unroll
  for (int c = 0; c < 16; ++c) sum = ln_add4(sum, v[c].x, v[c].y, v[c].z, v[c].w);
  const float mean = sum * (1.0f / 128.0f);
  const float2 mm = make_float2(-mean, -mean);
#pragma unroll
  for (int c = 0; c < 16; ++c) sq = ln_square(ln_square(ln_square(ln_square(sq, v[c].x, mm), v[c].y, mm), v[c].z, mm), v[c].w, mm);
  const float rstd = rsqrtf(sq * (1.0f / 128.0f) + eps);
  const float2 rr = make_float2(rstd, rstd);
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    const uint4 g = reinterpret_cast<const uint4*>(gamma2)[c], b = reinterpret_cast<const uint4*>(beta2)[c];
    v[c] = make_uint4(ln_affine(v[c].x, mm, rr, g.x, b.x), ln_affine(v[c].y, mm, rr, g.y, b.y),
                      ln_affine(v[c].z, mm, rr, g.z, b.z), ln_affine(v[c].w, mm, rr, g.w, b.w));
  }
}
// v[0..7] = slab 0 chunks, v[8..15] = slab 1 chunks (16 bytes = 8 channels each).
__device__ __forceinline__ void ln_load_row(const uint8_t* tile, int row, uint4 (&v)[16]) {
#pragma unroll
  for (int c = 0; c < 16; ++c) v[c] = *reinterpret_cast<const uint4*>(tile + (c >> 3) * SLAB_BYTES + sw128_offset(row, c & 7));
}
__device__ __forceinline__ void ln_store_row(uint8_t* tile, int row, const uint4 (&v)[16]) {
#pragma unroll
  for (int c = 0; c < 16; ++c) *reinterpret_cast<uint4*>(tile + (c >> 3) * SLAB_BYTES + sw128_offset(row, c & 7)) = v[c];
}

// The same layer norm (the same bits) as three sweeps over the row in shared memory - mean,
// variance, normalise - holding UNROLL words of 16 bytes at a time instead of the whole row: for
// kernels whose other roles leave the layer-norm warps few registers.
template <int UNROLL>
__device__ __forceinline__ void ln_row_sweeps(uint8_t* tile, int row, const uint32_t* gamma2, const uint32_t* beta2,
                                              float eps) {
  float sum = 0.f, sq = 0.f;
#pragma unroll UNROLL
  for (int c = 0; c < 16; ++c) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile + (c >> 3) * SLAB_BYTES + sw128_offset(row, c & 7));
    sum = ln_add4(sum, v.x, v.y, v.z, v.w);
  }
  const float mean = sum * (1.0f / 128.0f);
  const float2 mm = make_float2(-mean, -mean);
#pragma unroll UNROLL
  for (int c = 0; c < 16; ++c) {
    const uint4 v = *reinterpret_cast<const uint4*>(tile + (c >> 3) * SLAB_BYTES + sw128_offset(row, c & 7));
    sq = ln_square(ln_square(ln_square(ln_square(sq, v.x, mm), v.y, mm), v.z, mm), v.w, mm);
  }
  const float rstd = rsqrtf(sq * (1.0f / 128.0f) + eps);
  const float2 rr = make_float2(rstd, rstd);
#pragma unroll UNROLL
  for (int c = 0; c < 16; ++c) {
    uint4* ptr = reinterpret_cast<uint4*>(tile + (c >> 3) * SLAB_BYTES + sw128_offset(row, c & 7));
    const uint4 v = *ptr, g = reinterpret_cast<const uint4*>(gamma2)[c], b = reinterpret_cast<const uint4*>(beta2)[c];
    *ptr = make_uint4(ln_affine(v.x, mm, rr, g.x, b.x), ln_affine(v.y, mm, rr, g.y, b.y), ln_affine(v.z, mm, rr, g.z, b.z),
                      ln_affine(v.w, mm, rr, g.w, b.w));
  }
}

// Two threads per row: lanes l and l ^ 16 of a warp share row (l & 15) of the warp's 16
// rows; `half` = l >> 4 takes the 64 channels of slab `half`, and the two partial sums
// meet through one shuffle each. Half the instructions and half the dependency chain
// per thread, and twice the warps: the layer norm is what a projection tile waits for.
// Must be called by all 32 lanes of the warp. Same rounding points as ln_row_words;
// the fp32 statistics are summed in a different order (four partial sums per thread).
__device__ __forceinline__ void ln_row_two_threads(uint8_t* tile, int row, int half, const uint32_t* gamma2,
                                                   const uint32_t* beta2, float eps) {
  uint4 v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const uint4*>(tile + half * SLAB_BYTES + sw128_offset(row, c));
  float2 s[2] = {}, q[2] = {};  // the four partial sums: words 0, 1 | 2, 3 of each chunk
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    s[0] = __fadd2_rn(s[0], make_float2(sum_bf16x2(v[c].x), sum_bf16x2(v[c].y)));
    s[1] = __fadd2_rn(s[1], make_float2(sum_bf16x2(v[c].z), sum_bf16x2(v[c].w)));
  }
  float sum = (s[0].x + s[0].y) + (s[1].x + s[1].y);
  sum += __shfl_xor_sync(0xffffffffu, sum, 16);
  const float mean = sum * (1.0f / 128.0f);
  const float2 mm = make_float2(-mean, -mean);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float2 d0 = add_bf16x2(mm, w[2 * u]), d1 = add_bf16x2(mm, w[2 * u + 1]);
      const float2 a = make_float2(d0.x, d1.x), b = make_float2(d0.y, d1.y);
      q[u] = __ffma2_rn(b, b, __ffma2_rn(a, a, q[u]));
    }
  }
  float sq = (q[0].x + q[0].y) + (q[1].x + q[1].y);
  sq += __shfl_xor_sync(0xffffffffu, sq, 16);
  const float rstd = rsqrtf(sq * (1.0f / 128.0f) + eps);
  const float2 rr = make_float2(rstd, rstd);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint4 g = reinterpret_cast<const uint4*>(gamma2)[half * 8 + c], b = reinterpret_cast<const uint4*>(beta2)[half * 8 + c];
    *reinterpret_cast<uint4*>(tile + half * SLAB_BYTES + sw128_offset(row, c)) =
        make_uint4(ln_affine(v[c].x, mm, rr, g.x, b.x), ln_affine(v[c].y, mm, rr, g.y, b.y),
                   ln_affine(v[c].z, mm, rr, g.z, b.z), ln_affine(v[c].w, mm, rr, g.w, b.w));
  }
}

}  // namespace b200
