// Triangle attention, projection stage.
//
//   xn   = LN(x)                                   (x is read through caller strides,
//                                                   so the ending node is the same
//                                                   kernel on swapped strides)
//   q    = bf16(bf16(xn @ Wq) / bf16(sqrt(32)))    [o][t][128]   heads-major channels
//   k    = bf16(xn @ Wk)                            [o][t][128]
//   vT   = fp16(bf16(xn @ Wv))                      [o][128][ld]  channel-major per row o
//   bias = bf16(xn @ Wb)                            [4][o][ld]    (tri_bias[h][j][k] of the
//                                                   reference with j = o, k = t)
//
// Reference: src/foldjax/models/boltz2/models/triangle/triangle_attention.py
// :132 (LN), :144-146 (bias), :360-382 (fused projections), :399-400 (q scale).
// The gate projection is not done here: the output stage recomputes it from x,
// which costs the same bytes as reading a stored gate and saves writing one.
//
// V is stored transposed and in fp16: the core kernel multiplies P (fp16, 11
// significand bits) by V on the tensor cores. A bf16-rounded value of magnitude in
// [2^-14, 65504] is exactly representable in fp16 (8 significand bits fit in 11); larger
// ones saturate, values in [2^-24, 2^-14) land on fp16 subnormals and lose significand
// bits (at most the absolute 2^-25), smaller ones flush to zero. V is a layer-normed
// projection of order one, so only the exact range matters in practice.
//
// One tile = 128 consecutive pairs (o, t0..t0+127). Persistent, one CTA per SM:
//   warp 0      TMA producer (weights once, x tiles in a 2-stage ring)
//   warp 1      MMA issuer: [q|k] = xn.[Wq|Wk]^T (N=256), bias = xn.Wb^T (N=16),
//               vT = Wv.xn^T ("transposed": a TMEM lane is a channel)
//   warps 2-9   layer norm in place (two threads per pair)
//   warps 10-17 epilogue: one warpgroup per 64 channels of q and k and per 64 pairs of vT, each
//               with a staging slab, of which a warp fills and stores 32 rows
// TMEM: [q|k] 256 columns, vT 128, bias 16; each group is released on its own
// so the next tile's MMAs overlap this tile's epilogue.
// Bound: HBM (read x, write q, k, vT: 4 * n*n*128*2 bytes). By events around the launch, n = 200 / 512 / 1003:
// 19.0 / 54.5 / 187 us with a store per warpgroup, behind two barriers and the read of the store before;
// 16.9 / 52.0 / 183 with one per warp, whose read is waited for while the accumulators are fetched.
#include <cuda_fp16.h>

#include "host.cuh"
#include "ln.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int XSTAGES = 2;
constexpr int TILE_BYTES = 2 * SLAB_BYTES;
constexpr int W_BYTES = 6 * SLAB_BYTES;  // Wq, Wk, Wv: two boxes [128 in][64 out] each, MN-major
constexpr int WB_SLAB = 16 * 128;        // Wb, K-major: [16 heads (4 used)][64 in], two slabs
constexpr int LN_WARPS = 8, EPI_WARPS = 8;
constexpr int THREADS = 64 + (LN_WARPS + EPI_WARPS) * 32;
constexpr uint32_t TM_QK = 0, TM_V = 256, TM_B = 384;
enum { G_QK = 0, G_B = 1, G_V = 2 };

struct Smem {
  uint8_t w[W_BYTES];
  uint8_t wb[2 * WB_SLAB];
  uint8_t x[XSTAGES][TILE_BYTES];
  uint8_t out[TILE_BYTES];  // staging, one 16 KiB slab per epilogue warpgroup (q, then k, then vT)
  alignas(16) uint32_t gamma2[64], beta2[64];
  uint64_t w_full, x_full[XSTAGES], xn_full[XSTAGES], x_empty[XSTAGES], acc_full[3], acc_empty[3];
  uint32_t tmem_base;
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

struct Params {
  int n_outer, n_inner, tiles_inner;
  uint32_t total_tiles;
  const void* gamma;
  const void* beta;
  const __nv_bfloat16* w_bias;  // [128][4]
  bool early_weights;           // the weights may be read before pdl_wait()
  MaskBiasOut mb;               // mb.out null: no mask-bias rows wanted
  __nv_bfloat16* bias;
  long long ld;           // pitch of bias rows (elements)
  long long bias_head_stride;
  float q_scale;          // bf16(sqrt(head_dim))
  float eps;
  int* status;
};

__global__ void __launch_bounds__(THREADS, 1)
att_project_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_wq,
                   const __grid_constant__ CUtensorMap tm_wk, const __grid_constant__ CUtensorMap tm_wv,
                   const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_vt,
                   const Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  // (through a shuffle, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  if ((smem_u32(smem_raw) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicCAS(p.status, ST_OK, 900);
    return;
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_wq);
    tma_prefetch_desc(&tm_wk);
    tma_prefetch_desc(&tm_wv);
    mbar_init(&sm.w_full, 1);
    for (int s = 0; s < XSTAGES; ++s) {
      mbar_init(&sm.x_full[s], 1);
      mbar_init(&sm.xn_full[s], LN_WARPS);
      mbar_init(&sm.x_empty[s], 1);
    }
    for (int g = 0; g < 3; ++g) {
      mbar_init(&sm.acc_full[g], 1);
      mbar_init(&sm.acc_empty[g], g == G_B ? 4 : EPI_WARPS);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  if (!p.early_weights) pdl_wait();
  if (threadIdx.x >= 64 && threadIdx.x < 128) {
    sm.gamma2[threadIdx.x - 64] = ln_param_pair(p.gamma, threadIdx.x - 64);
    sm.beta2[threadIdx.x - 64] = ln_param_pair(p.beta, threadIdx.x - 64);
  }
  for (int idx = threadIdx.x; idx < 2 * 16 * 64; idx += THREADS) {  // (slab, head, channel of the slab)
    const int slab = idx >> 10, row = (idx >> 6) & 15, c = idx & 63;
    const __nv_bfloat16 v = row < 4 ? p.w_bias[(slab * 64 + c) * 4 + row] : __float2bfloat16_rn(0.f);
    *reinterpret_cast<__nv_bfloat16*>(sm.wb + slab * WB_SLAB + sw128_offset(row, c >> 3) + (c & 7) * 2) = v;
  }
  fence_proxy_async();
  if (warp == 0 && lane == 0) {  // (the thread that initialised the barrier)
    mbar_expect_tx(&sm.w_full, W_BYTES);
    for (int g = 0; g < 3; ++g)
      for (int s = 0; s < 2; ++s)
        tma_load_2d(sm.w + (g * 2 + s) * SLAB_BYTES, g == 0 ? &tm_wq : g == 1 ? &tm_wk : &tm_wv, &sm.w_full, s * 64, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;
  int status = -1;

  // (32-bit: a 64-bit division costs a role hundreds of cycles per tile)
  auto locate = [&](uint32_t tile, int& o, int& t0) {
    const uint32_t q = tile / static_cast<uint32_t>(p.tiles_inner);
    o = q;
    t0 = (tile - q * p.tiles_inner) * 128;
  };
  auto load_x = [&](int stage, int o, int t0) {
    mbar_expect_tx(&sm.x_full[stage], TILE_BYTES);
    tma_load_3d(sm.x[stage], &tm_x, &sm.x_full[stage], 0, t0, o);
    tma_load_3d(sm.x[stage] + SLAB_BYTES, &tm_x, &sm.x_full[stage], 64, t0, o);
  };
  int first_o, first_t0;  // the first tile, located ahead of the wait and requested right behind it
  locate(blockIdx.x, first_o, first_t0);
  if (p.early_weights) pdl_wait();
  if (threadIdx.x == 0) load_x(0, first_o, first_t0);
  pdl_trigger();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 1;  // (stage 0 has the first tile)
      uint32_t phase = 0;
      for (uint32_t tile = blockIdx.x + gridDim.x; tile < p.total_tiles; tile += gridDim.x) {
        int o, t0;
        locate(tile, o, t0);
        if (!mbar_wait(&sm.x_empty[stage], phase ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
        load_x(stage, o, t0);
        if (++stage == XSTAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 128) | UMMA_B_MN;
      constexpr uint32_t idesc_b = umma_idesc_bf16(128, 16);
      constexpr uint32_t idesc_v = umma_idesc_bf16(128, 128) | UMMA_A_MN;
      bool alive = mbar_wait(&sm.w_full, 0, p.status, ST_TIMEOUT_MMA);
      int stage = 0;
      uint32_t phase = 0, it = 0;
      for (uint32_t tile = blockIdx.x; tile < p.total_tiles && alive; tile += gridDim.x, ++it) {
        if (!mbar_wait(&sm.xn_full[stage], phase, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t xs = smem_u32(sm.x[stage]);
        const uint32_t ws = smem_u32(sm.w);
        // [q|k]: A = xn (rows = pairs), B = Wq, Wk
        if (!mbar_wait(&sm.acc_empty[G_QK], (it & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint64_t bdesc = umma_desc_mnmajor(ws + half * 2 * SLAB_BYTES, SLAB_BYTES);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_bf16_ss(tmem_base + TM_QK + half * 128,
                         umma_desc_advance(umma_desc_kmajor(xs + (k >> 2) * SLAB_BYTES, 128), (k & 3) * 32),
                         umma_desc_advance(bdesc, k * 2048), idesc_qk, k != 0);
        }
        umma_commit(&sm.acc_full[G_QK]);
        // bias: A = xn, B = Wb, N = 16
        if (!mbar_wait(&sm.acc_empty[G_B], (it & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const uint64_t adesc = umma_desc_kmajor(xs + s * SLAB_BYTES, 128);
          const uint64_t bdesc = umma_desc_kmajor(smem_u32(sm.wb) + s * WB_SLAB, 128);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ss(tmem_base + TM_B, umma_desc_advance(adesc, k * 32), umma_desc_advance(bdesc, k * 32),
                         idesc_b, (s | k) != 0);
        }
        umma_commit(&sm.acc_full[G_B]);
        // vT: A = Wv (rows = channels), B = xn (rows = pairs)
        if (!mbar_wait(&sm.acc_empty[G_V], (it & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint64_t vdesc = umma_desc_mnmajor(ws + 4 * SLAB_BYTES, SLAB_BYTES);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + TM_V, umma_desc_advance(vdesc, k * 2048),
                       umma_desc_advance(umma_desc_kmajor(xs + (k >> 2) * SLAB_BYTES, 128), (k & 3) * 32), idesc_v, k != 0);
        umma_commit(&sm.acc_full[G_V]);
        umma_commit(&sm.x_empty[stage]);
        if (++stage == XSTAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp < 2 + LN_WARPS) {
    const int r = (warp - 2) * 16 + (lane & 15);  // pair of the tile; lanes l and l ^ 16 share it
    int stage = 0;
    uint32_t phase = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x) {
      if (p.mb.out && lane < 16) {  // the core's mask-bias row of these pairs, pitch padding included
        int o, t;
        locate(tile, o, t);
        t += r;
        if (t < p.mb.ld)
          p.mb.out[static_cast<long long>(o) * p.mb.ld + t] =
              t >= p.n_inner ? -INFINITY
              : p.mb.mask    ? mask_bias(p.mb.mask[o * p.mb.ms_outer + t * p.mb.ms_inner], p.mb.inf, false)
                             : 0.0f;
      }
      if (!mbar_wait(&sm.x_full[stage], phase, p.status, ST_TIMEOUT_PROLOGUE)) break;
      __syncwarp();
      ln_row_two_threads(sm.x[stage], r, lane >> 4, sm.gamma2, sm.beta2, p.eps);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.xn_full[stage]);
      if (++stage == XSTAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else {
    const int quarter = warp & 3, group = (warp - 2 - LN_WARPS) >> 2;
    const int row = quarter * 32 + lane;  // TMEM lane: a pair for q/k/bias, a channel for vT
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    uint8_t* out = sm.out + group * SLAB_BYTES;
    const uint32_t qs = pack_bf16x2(p.q_scale, p.q_scale);
    const float q_inv = 1.0f / bf16_lo(qs);
    uint32_t it = 0;
    // (a vote: TMEM accesses take the whole warp. Each warp stages and stores its own 32 rows)
    auto acc_wait = [&](int g) {
      return __all_sync(0xffffffffu, mbar_wait(&sm.acc_full[g], it & 1, p.status, ST_TIMEOUT_EPILOGUE));
    };
    auto rows_free = [&] {  // the warp's previous store has read them: asked when there is something to go there
      if (lane == 0) tma_store_wait_read();
      __syncwarp();
    };
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x, ++it) {
      int o, t0;
      locate(tile, o, t0);
      // ---- q and k: thread = pair, 64 channels of each
      if (!acc_wait(G_QK)) break;
      tc_fence_after();
#pragma unroll 1
      for (int part = 0; part < 2; ++part) {  // q, then k
#pragma unroll
        for (int c2 = 0; c2 < 2; ++c2) {
          uint32_t r[32];
          tmem_ld32(lane_addr + TM_QK + part * 128 + group * 64 + c2 * 32, r);
          if (c2 == 0) rows_free();
          tmem_ld_wait();
#pragma unroll
          for (int g4 = 0; g4 < 4; ++g4) {
            uint32_t u[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              uint32_t v2 = pack_bf16x2(__uint_as_float(r[8 * g4 + 2 * e]), __uint_as_float(r[8 * g4 + 2 * e + 1]));
              // q / sqrt(d) as the product with the rounded reciprocal: the same bf16 as the true
              // division for every bf16 q (the quotient is never within 1e-5 of a rounding boundary)
              if (part == 0) v2 = pack_bf16x2(bf16_lo(v2) * q_inv, bf16_hi(v2) * q_inv);
              u[e] = v2;
            }
            // row = pair, 16-byte chunk = 8 channels
            *reinterpret_cast<uint4*>(out + sw128_offset(row, c2 * 4 + g4)) = make_uint4(u[0], u[1], u[2], u[3]);
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && t0 + quarter * 32 < p.n_inner) {  // pairs past n_inner are outside the tensor and are not written
          tma_store_3d(part ? &tm_k : &tm_q, out + quarter * 4096, group * 64, t0 + quarter * 32, o);
          tma_store_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.acc_empty[G_QK]);
      if (group == 0) {  // ---- bias: thread = pair, 4 heads
        if (!acc_wait(G_B)) break;
        tc_fence_after();
        uint32_t r[16];
        tmem_ld16(lane_addr + TM_B, r);
        tmem_ld_wait();
        const int t = t0 + row;
        if (t < p.n_inner) {
#pragma unroll
          for (int h = 0; h < 4; ++h)
            p.bias[h * p.bias_head_stride + static_cast<long long>(o) * p.ld + t] =
                __float2bfloat16_rn(__uint_as_float(r[h]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acc_empty[G_B]);
      }
      // ---- vT: thread = channel, 64 pairs -> one contiguous run of the row
      if (!acc_wait(G_V)) break;
      tc_fence_after();
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {
        uint32_t r[32];
        tmem_ld32(lane_addr + TM_V + group * 64 + c2 * 32, r);
        if (c2 == 0) rows_free();
        tmem_ld_wait();
#pragma unroll
        for (int g4 = 0; g4 < 4; ++g4) {
          uint32_t u[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = 8 * g4 + 2 * e;
            const uint32_t b2 = pack_bf16x2(__uint_as_float(r[c]), __uint_as_float(r[c + 1]));  // bf16(xn @ Wv)
            const __half2 h2 = __floats2half2_rn(bf16_lo(b2), bf16_hi(b2));
            u[e] = *reinterpret_cast<const uint32_t*>(&h2);
          }
          // row = channel, 16-byte chunk = 8 pairs
          *reinterpret_cast<uint4*>(out + sw128_offset(row, c2 * 4 + g4)) = make_uint4(u[0], u[1], u[2], u[3]);
        }
      }
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && t0 + group * 64 < p.n_inner) {
        tma_store_3d(&tm_vt, out + quarter * 4096, t0 + group * 64, quarter * 32, o);
        tma_store_commit();
      }
      if (lane == 0) mbar_arrive(&sm.acc_empty[G_V]);
    }
    status = stores_read_and_status(lane == 0, p.status);
  }

  settle(status, p.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace
}  // namespace b200

extern "C" size_t b200tri_triatt_project_workspace_bytes(void) { return 512 * 128 * 2 + 1024; }

extern "C" int b200tri_triatt_project(const b200tri_triatt_project_args* a, b200tri_stream_t stream) {
  return b200::att_project_launch(a, nullptr, reinterpret_cast<cudaStream_t>(stream));
}

int b200::att_project_launch(const b200tri_triatt_project_args* a, const MaskBiasOut* mb, cudaStream_t stream) {
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "att project: null args");
  B200_REQUIRE(a->x && a->q && a->k && a->vt && a->bias && a->norm_scale && a->norm_bias && a->w_q && a->w_k &&
                   a->w_v && a->w_bias,
               B200TRI_ERR_INVALID, "att project: null pointer argument");
  B200_REQUIRE(a->n_outer > 0 && a->n_inner > 0, B200TRI_ERR_INVALID, "att project: sizes must be positive");
  B200_REQUIRE(a->heads == 4 && a->head_dim == 32, B200TRI_ERR_UNSUPPORTED,
               "att project: built for 4 heads x 32 (got %d x %d)", a->heads, a->head_dim);
  B200_REQUIRE(a->xs_outer % 8 == 0 && a->xs_inner % 8 == 0 && a->ld % 8 == 0 && a->ld >= a->n_inner,
               B200TRI_ERR_INVALID, "att project: strides/pitch must be multiples of 8 elements, ld >= n_inner");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(a->q) | reinterpret_cast<uintptr_t>(a->k) |
                 reinterpret_cast<uintptr_t>(a->vt) | reinterpret_cast<uintptr_t>(a->bias)) & 15) == 0,
               B200TRI_ERR_INVALID, "att project: outputs must be 16-byte aligned");
  B200_REQUIRE(a->workspace && a->workspace_bytes >= b200tri_triatt_project_workspace_bytes(), B200TRI_ERR_WORKSPACE,
               "att project: workspace of %zu bytes needed", b200tri_triatt_project_workspace_bytes());
  int* status = device_status_word();
  B200_REQUIRE(status != nullptr, B200TRI_ERR_CUDA, "att project: no current CUDA device");

  // the weights are read in place; the workspace is only for one that is not 16-byte aligned
  Carver ws(a->workspace);
  const void* const w_in[3] = {a->w_q, a->w_k, a->w_v};
  const void* w[3];
  bool in_place = true;
  for (int i = 0; i < 3; ++i) {
    const int rc = aligned_weight(w_in[i], 128 * 128 * 2, ws.take<__nv_bfloat16>(128 * 128), stream, &w[i]);
    if (rc) return rc;
    in_place = in_place && w[i] == w_in[i];
  }
  CUtensorMap tm_x, tm_w[3], tm_q, tm_k, tm_vt;
  {  // q and k [n_outer][n_inner][128], written as tiles of [32 pairs][64 channels]
    const uint64_t dims[3] = {128, (uint64_t)a->n_inner, (uint64_t)a->n_outer};
    const uint64_t str[2] = {256, (uint64_t)a->n_inner * 256};
    const uint32_t box[3] = {64, 32, 1};
    int rc = make_tmap(&tm_q, a->q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
    rc = make_tmap(&tm_k, a->k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {  // vT [n_outer][128][ld] fp16, written as tiles of [32 channels][64 pairs]
    const uint64_t dims[3] = {(uint64_t)a->n_inner, 128, (uint64_t)a->n_outer};
    const uint64_t str[2] = {(uint64_t)a->ld * 2, (uint64_t)a->ld * 2 * 128};
    const uint32_t box[3] = {64, 32, 1};
    int rc = make_tmap(&tm_vt, a->vt, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    const uint64_t dims[3] = {128, (uint64_t)a->n_inner, (uint64_t)a->n_outer};
    const uint64_t str[2] = {(uint64_t)a->xs_inner * 2, (uint64_t)a->xs_outer * 2};
    const uint32_t box[3] = {64, 128, 1};
    int rc = make_tmap(&tm_x, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  for (int i = 0; i < 3; ++i) {
    const int rc = make_weight_map(&tm_w[i], w[i], 128, 128, 128);
    if (rc) return rc;
  }
  Params p;
  p.n_outer = a->n_outer;
  p.n_inner = a->n_inner;
  p.tiles_inner = (a->n_inner + 127) / 128;
  const long long tiles = static_cast<long long>(p.tiles_inner) * a->n_outer;
  B200_REQUIRE(tiles < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "att project: too many tiles (%lld)", tiles);
  p.total_tiles = static_cast<uint32_t>(tiles);
  p.gamma = a->norm_scale;
  p.beta = a->norm_bias;
  p.w_bias = static_cast<const __nv_bfloat16*>(a->w_bias);
  p.early_weights = pdl_chained() && in_place;
  p.mb = mb ? *mb : MaskBiasOut{};
  p.bias = static_cast<__nv_bfloat16*>(a->bias);
  p.ld = a->ld;
  p.bias_head_stride = a->bias_head_stride;
  p.q_scale = __bfloat162float(__float2bfloat16_rn(sqrtf(static_cast<float>(a->head_dim))));
  p.eps = a->eps;
  p.status = status;

  {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(att_project_kernel), (int)sizeof(Smem));
    if (rc) return rc;
  }
  const long long grid = tiles < sm_count() ? tiles : sm_count();
  {
    TimedLaunch timed(K_TRIATT_PROJECT, stream);
    return launch(att_project_kernel, dim3(static_cast<unsigned>(grid)), dim3(THREADS), sizeof(Smem), stream, true, tm_x,
                  tm_w[0], tm_w[1], tm_w[2], tm_q, tm_k, tm_vt, p);
  }
}
