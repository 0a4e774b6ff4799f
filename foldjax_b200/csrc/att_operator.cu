// The attention-core operator: q, k, v and the result in the caller's [I][H][token][D] order.
//
// Reference: the signature core(q, k, v, tri_bias, mask_bias), pallas_attention_core,
// src/foldjax/models/boltz2/models/triangle/triangle_attention_pallas.py:180.
//
// Queries, keys and the result need no relayout: they are 4-D tensor maps (channel, head, token,
// row) for the core. What the core cannot read in place is prepared by one kernel: V transposed
// to fp16 [row][head * 32 + d][key], and the mask-bias rows. The pair bias is read where it is
// unless its rows are off the 16-byte grid TMA needs, or float32.
//
// Bound of the preparation: memory, 2 + 2 bytes per element of V. 4 heads x 384 x 384 x 32: 97 us with the core (this and the
// next: calls replayed in a row on the same operands); relayout copies of all five operands alone are 250. Small operators are
// launches: with the bias rows in one of their own 60 / 100 / 203 / 300 tokens took 10.3 / 12.4 / 33.7 / 76.2 us, 7.9 / 10.9 / 28.4 / 70.6 so
// (the core's last step of its own width among it).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "host.cuh"
#include "tc.cuh"

namespace b200 {
namespace {

constexpr int HEADS = 4, D = 32, KT = 64;
constexpr int PITCH = KT + 2;  // halves per channel row of the transposed tile: conflict-free both ways

struct Chunk {  // 8 channels of one key
  float f[8];
};
__device__ __forceinline__ Chunk load_chunk(const __nv_bfloat16* p) {
  const uint4 w = *reinterpret_cast<const uint4*>(p);
  return {bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y), bf16_lo(w.z), bf16_hi(w.z), bf16_lo(w.w), bf16_hi(w.w)};
}
__device__ __forceinline__ Chunk load_chunk(const float* p) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  return {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

// One block per (row, 64 keys): all four heads, so that every thread has four loads in flight. Behind those blocks, where the pair
// bias [4 * n_j][n_k] is to be copied to bf16 rows of pitch ld, one per eight of its rows.
struct BiasCopy {
  const void* src;  // or null
  __nv_bfloat16* dst;
  long long rows;
};
template <typename T, typename B>
__global__ void __launch_bounds__(256)
prepare_kernel(const T* __restrict__ v, const float* __restrict__ mask, __half* __restrict__ vt, float* __restrict__ mb,
               int n_k, int ld, unsigned blocks, const BiasCopy bias, bool chained) {
  __shared__ __half tile[HEADS][D][PITCH];
  if (chained) {
    pdl_wait();
    pdl_trigger();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (blockIdx.x >= blocks) {
    const long long r = static_cast<long long>(blockIdx.x - blocks) * 8 + warp;
    if (r >= bias.rows) return;
    const B* src = static_cast<const B*>(bias.src) + r * n_k;
    __nv_bfloat16* dst = bias.dst + r * ld;
    // (sixteen loads of a thread in flight, two neighbours stored at a time: with four, one element at a time, the whole preparation of
    // 64 rows x 1003 keys took 20.1 us, 25.5 with a float32 bias, 10.7 and 10.4 so; of 16 x 2048, float32, 42 and 19, of 8 x 3001 80 / 105
    // and 31 / 34, 2 x 515 4.8 and 3.0; 203 x 203 6.3 / 7.0 and 5.9)
    for (int k0 = 2 * lane; k0 < ld; k0 += 512) {
      float f[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int k = k0 + 64 * (u / 2) + u % 2;
        f[u] = k < n_k ? static_cast<float>(src[k]) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)  // (ld is a multiple of 64)
        if (k0 + 64 * u < ld) *reinterpret_cast<uint32_t*>(dst + k0 + 64 * u) = pack_bf16x2(f[2 * u], f[2 * u + 1]);
    }
    return;
  }
  const int tiles = ld / KT;
  const int i = blockIdx.x / tiles, k0 = (blockIdx.x - i * tiles) * KT;
  const int key = threadIdx.x >> 2, c = (threadIdx.x & 3) * 8;
  const bool valid = k0 + key < n_k;
  const T* src = v + (static_cast<long long>(i) * HEADS * n_k + k0 + key) * D + c;
  Chunk x[HEADS];
#pragma unroll
  for (int h = 0; h < HEADS; ++h) x[h] = valid ? load_chunk(src + static_cast<long long>(h) * n_k * D) : Chunk{};
#pragma unroll
  for (int h = 0; h < HEADS; ++h)
#pragma unroll
    for (int e = 0; e < 8; ++e) tile[h][c + e][key] = __float2half_rn(x[h].f[e]);
  if (threadIdx.x < KT) {
    const int k = k0 + threadIdx.x;
    mb[static_cast<long long>(i) * ld + k] =
        k < n_k ? mask_bias(mask[static_cast<long long>(i) * n_k + k], 0.f, true) : -INFINITY;
  }
  __syncthreads();
  __half* dst = vt + static_cast<long long>(i) * HEADS * D * ld + k0;
  for (int r = warp; r < HEADS * D; r += 8)
    reinterpret_cast<uint32_t*>(dst + static_cast<long long>(r) * ld)[lane] =
        reinterpret_cast<const uint32_t*>(&tile[r / D][r % D][0])[lane];
}

struct Plan {
  size_t mb, vt, bias, total;
};
Plan plan(int n_i, int n_j, int n_k) {
  Plan p;
  const size_t ld = round_up(n_k, KT);
  auto up = [](size_t x) { return (x + 1023) / 1024 * 1024; };
  p.mb = 0;
  p.vt = up(b200tri_triatt_core_workspace_bytes(n_i, n_k));
  p.bias = p.vt + up(static_cast<size_t>(n_i) * HEADS * D * ld * 2);
  p.total = p.bias + up(static_cast<size_t>(HEADS) * n_j * ld * 2);
  return p;
}

}  // namespace
}  // namespace b200

extern "C" size_t b200tri_attention_core_workspace_bytes(int32_t n_i, int32_t n_j, int32_t n_k) {
  if (n_i <= 0 || n_j <= 0 || n_k <= 0) return 0;
  return b200::plan(n_i, n_j, n_k).total;
}

extern "C" int b200tri_attention_core(const b200tri_attention_core_args* a, b200tri_stream_t stream_) {
  using namespace b200;
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "attention core: null args");
  B200_REQUIRE(a->batch > 0 && a->n_i > 0 && a->n_j > 0 && a->n_k > 0, B200TRI_ERR_INVALID,
               "attention core: sizes must be positive");
  B200_REQUIRE(a->heads == HEADS && a->head_dim == D, B200TRI_ERR_UNSUPPORTED,
               "attention core: built for 4 heads x 32 (got %d x %d)", a->heads, a->head_dim);
  B200_REQUIRE(a->q && a->k && a->v && a->bias && a->mask_bias && a->out, B200TRI_ERR_INVALID,
               "attention core: null pointer argument");
  const uintptr_t bases = reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) |
                          reinterpret_cast<uintptr_t>(a->v) | reinterpret_cast<uintptr_t>(a->out);
  B200_REQUIRE((bases & 15) == 0, B200TRI_ERR_INVALID, "attention core: q, k, v and out must be 16-byte aligned");
  const Plan pl = plan(a->n_i, a->n_j, a->n_k);
  B200_REQUIRE(a->workspace && a->workspace_bytes >= pl.total, B200TRI_ERR_WORKSPACE,
               "attention core: workspace of %zu bytes needed, got %zu", pl.total, a->workspace_bytes);
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a->workspace) & 1023) == 0, B200TRI_ERR_INVALID,
               "attention core: workspace must be 1024-byte aligned");
  const int ld = round_up(a->n_k, KT);
  const long long blocks = static_cast<long long>(a->n_i) * (ld / KT);
  B200_REQUIRE(blocks < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "attention core: too many rows times keys for one launch");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  uint8_t* ws = static_cast<uint8_t*>(a->workspace);
  float* mb = reinterpret_cast<float*>(ws + pl.mb);
  __half* vt = reinterpret_cast<__half*>(ws + pl.vt);
  const bool bias_in_place = !a->bias_f32 && a->n_k % 8 == 0 && (reinterpret_cast<uintptr_t>(a->bias) & 15) == 0;
  const size_t tok_j = static_cast<size_t>(a->n_i) * HEADS * a->n_j * D, tok_k = static_cast<size_t>(a->n_i) * HEADS * a->n_k * D;
  const size_t bias_elems = static_cast<size_t>(HEADS) * a->n_j * a->n_k;
  const CoreStrides strides = {D, static_cast<long long>(a->n_j) * D, static_cast<long long>(a->n_k) * D,
                               static_cast<long long>(a->n_j) * D * HEADS, static_cast<long long>(a->n_k) * D * HEADS};
  const long long bias_rows = bias_in_place ? 0 : static_cast<long long>(HEADS) * a->n_j;
  const long long grid_blocks = blocks + (bias_rows + 7) / 8;
  B200_REQUIRE(grid_blocks < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "attention core: too many rows times keys for one launch");
  // Programmatic launches from the kernel before to the core, where no SM has two blocks of the preparation: the core's
  // CTA has room beside one (48 / 60 / 64 tokens 8.3 / 8.8 / 8.4 us without, 6.8 / 7.8 / 7.5 with; beside two it has not,
  // 77 / 88 / 100 tokens 9.8 / 10.6 / 10.7 and 10.0 / 12.7 / 13.6).
  const bool chained = grid_blocks <= sm_count();
  for (int b = 0; b < a->batch; ++b) {
    const float* mask = a->mask_bias + static_cast<size_t>(b) * a->n_i * a->n_k;
    const uint8_t* bias = static_cast<const uint8_t*>(a->bias) + b * bias_elems * (a->bias_f32 ? 4 : 2);
    __nv_bfloat16* copy = reinterpret_cast<__nv_bfloat16*>(ws + pl.bias);
    const BiasCopy rows = {bias, copy, bias_rows};
    auto go = [&](auto kernel, auto* values) {
      return launch(kernel, dim3(static_cast<unsigned>(grid_blocks)), dim3(256), 0, stream, chained, values + b * tok_k, mask, vt, mb,
                    a->n_k, ld, static_cast<unsigned>(blocks), rows, chained);
    };
    const auto* v32 = static_cast<const float*>(a->v);
    const auto* v16 = static_cast<const __nv_bfloat16*>(a->v);
    int rc;
    if (a->v_f32)
      rc = a->bias_f32 ? go(prepare_kernel<float, float>, v32) : go(prepare_kernel<float, __nv_bfloat16>, v32);
    else
      rc = a->bias_f32 ? go(prepare_kernel<__nv_bfloat16, float>, v16) : go(prepare_kernel<__nv_bfloat16, __nv_bfloat16>, v16);
    if (rc) return rc;
    b200tri_triatt_core_args ca = {};
    ca.bias = bias_in_place ? static_cast<const void*>(bias) : copy;
    ca.bias_ld = bias_in_place ? a->n_k : ld;
    ca.bias_head_stride = ca.bias_ld * a->n_j;
    ca.n_i = a->n_i;
    ca.n_j = a->n_j;
    ca.n_k = a->n_k;
    ca.heads = HEADS;
    ca.head_dim = D;
    ca.q = static_cast<const __nv_bfloat16*>(a->q) + b * tok_j;
    ca.k = static_cast<const __nv_bfloat16*>(a->k) + b * tok_k;
    ca.vt = vt;
    ca.v_ld = ld;
    ca.o = static_cast<__nv_bfloat16*>(a->out) + b * tok_j;
    ca.workspace = mb;
    ca.workspace_bytes = pl.vt;
    if ((rc = att_core_launch_premasked(&ca, &strides, stream))) return rc;
  }
  return B200TRI_OK;
}
