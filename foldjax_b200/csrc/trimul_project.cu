// Triangle multiplicative update, projection stage.
//
//   xn     = LN_in(x)
//   [a|b]  = sigmoid(xn @ g_in) * (xn @ p_in) * mask        (256 channels)
//
// written channel-major (a[d][o][t], b[d][o][t]) so the contraction stage can
// feed both operands to the tensor cores K-major. Reference:
// src/foldjax/models/boltz2/models/triangle/triangle.py:78-102.
//
// One tile = 128 consecutive pairs (o, t0..t0+127). The products are issued
// "transposed" - D[channel][pair] = W[channel][:] . xn[pair][:] - so a TMEM
// lane is an output channel, and a warpgroup of the epilogue turns 32 pairs of
// all channels into a staged tile of the channel-major output.
//
// Persistent kernel, one CTA per SM:
//   warp 0       TMA producer: weights once (128 KiB, resident), x tiles in a 2-stage ring
//   warp 1       MMA issuer: 4 groups (p_a, g_a, p_b, g_b) of 128x128x128 per tile
//   warps 2-9    layer norm, in place in the tile TMA delivered (two threads per pair)
//   warps 10-25  epilogue: TMEM -> sigmoid gate -> mask -> bf16 -> shared memory -> TMA store,
//                32 pairs per warpgroup (stored by the threads themselves, each 64-byte run went to
//                another channel plane: 32 lines per instruction, and the L1 pipe was the bound)
// TMEM: four 128-column accumulators; the a-half and the b-half are released
// separately so the MMAs of the next tile overlap the epilogue of this one.
//
// Bound: HBM by the bytes (read x once, write a and b once: 3 * n*n*128*2 bytes, 123 us at n = 1024);
// in fact the MUFU unit, two operations for each of a pair's 256 sigmoids: 74 % busy over the 204 us
// of a launch at n = 1024 (213 with a warp index the compiler did not know to be uniform, 285 with one
// epilogue warpgroup that stored each thread's run directly). It is not the only bound: the epilogue warps are at it
// 94 % of the time and the layer norm's 83 %, and what takes work off the MUFU unit or brings the epilogue forward
// costs the others as much. Measured and not better, by events around the launch at n = 1003 (226 us): the
// sigmoids' reciprocals on the FMA pipe (two Newton steps, the same bf16 results; 237-245 for half of them, three
// quarters and all), a store per warp (241), the previous store's read waited for behind the first loads (241).
#include <type_traits>

#include "host.cuh"
#include "ln.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int XSTAGES = 2;
constexpr int TILE_BYTES = 2 * SLAB_BYTES;  // 32 KiB: 128 pairs x 128 channels bf16
constexpr int W_BYTES = 8 * SLAB_BYTES;     // 128 KiB: 4 groups x 2 K-slabs
constexpr int MASK_SLOTS = 4;
constexpr int LN_WARPS = 8, EPI_WARPS = 16;  // the sigmoids of a tile want many warps: see below
constexpr int THREADS = 64 + (LN_WARPS + EPI_WARPS) * 32;

struct Smem {
  uint8_t w[W_BYTES];  // group g (p_a, g_a, p_b, g_b): two boxes [128 in][64 out], MN-major
  uint8_t x[XSTAGES][TILE_BYTES];
  uint8_t out[4][SLAB_BYTES / 2];       // per epilogue warpgroup: [128 channels][32 pairs], 64-byte swizzle
  __nv_bfloat16 mask[MASK_SLOTS][128];  // mask.astype(bf16), as the reference casts it
  alignas(16) uint32_t gamma2[64], beta2[64];
  uint64_t w_full, x_full[XSTAGES], xn_full[XSTAGES], x_empty[XSTAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

struct ProjParams {
  int n_outer, n_inner, tiles_inner;
  uint32_t total_tiles;
  const float* mask;
  long long ms_outer, ms_inner;
  const void* gamma;
  const void* beta;
  bool early_weights;  // the weights may be read before pdl_wait()
  int rows_per_block;
  float eps;
  int* status;
};
struct RaggedParams : ProjParams {  // the outputs as the threads address them
  __nv_bfloat16 *a, *b;
  long long ld, chan_stride, block_stride;
};

// RAGGED: rows end inside 16 bytes and what lies behind them is not ours. TMA would write it, so the
// maps end at the last whole 16 bytes and the threads store the rest.
template <bool RAGGED>
__global__ void __launch_bounds__(THREADS, 1)
project_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_p,
               const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ CUtensorMap tm_a,
               const __grid_constant__ CUtensorMap tm_b,
               const typename std::conditional<RAGGED, RaggedParams, ProjParams>::type p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  // (through a shuffle, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  if ((smem_u32(smem_raw) & 1023u) != 0) {  // operand tiles need 1 KiB alignment
    if (threadIdx.x == 0) atomicCAS(p.status, ST_OK, 900);
    return;
  }

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_p);
    tma_prefetch_desc(&tm_g);
    mbar_init(&sm.w_full, 1);
    for (int s = 0; s < XSTAGES; ++s) {
      mbar_init(&sm.x_full[s], 1);
      mbar_init(&sm.xn_full[s], LN_WARPS);
      mbar_init(&sm.x_empty[s], 1);
    }
    for (int h = 0; h < 2; ++h) {
      mbar_init(&sm.acc_full[h], 1);
      mbar_init(&sm.acc_empty[h], EPI_WARPS);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  if (!p.early_weights) pdl_wait();
  LnParam ln_param;
  if (threadIdx.x >= 64 && threadIdx.x < 192) ln_param.request(threadIdx.x < 128 ? p.gamma : p.beta, threadIdx.x & 63);
  if (warp == 0 && lane == 0) {  // (the thread that initialised the barrier)
    mbar_expect_tx(&sm.w_full, W_BYTES);
    for (int g = 0; g < 4; ++g)
      for (int s = 0; s < 2; ++s)
        tma_load_2d(sm.w + (g * 2 + s) * SLAB_BYTES, (g & 1) ? &tm_g : &tm_p, &sm.w_full, (g >> 1) * 128 + s * 64, 0);
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
      constexpr uint32_t idesc = umma_idesc_bf16(128, 128) | UMMA_A_MN;
      bool alive = mbar_wait(&sm.w_full, 0, p.status, ST_TIMEOUT_MMA);
      int stage = 0;
      uint32_t phase = 0, it = 0;
      for (uint32_t tile = blockIdx.x; tile < p.total_tiles && alive; tile += gridDim.x, ++it) {
        if (!mbar_wait(&sm.xn_full[stage], phase, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t xs = smem_u32(sm.x[stage]);
        for (int half = 0; half < 2 && alive; ++half) {
          if (!mbar_wait(&sm.acc_empty[half], (it & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) {
            alive = false;
            break;
          }
          tc_fence_after();
          for (int g = 0; g < 2; ++g) {
            const int group = half * 2 + g;
            const uint32_t d_tmem = tmem_base + group * 128;
            const uint64_t wdesc = umma_desc_mnmajor(smem_u32(sm.w + group * 2 * SLAB_BYTES), SLAB_BYTES);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const uint64_t xdesc = umma_desc_kmajor(xs + (k >> 2) * SLAB_BYTES, 128);
              umma_bf16_ss(d_tmem, umma_desc_advance(wdesc, k * 2048), umma_desc_advance(xdesc, (k & 3) * 32), idesc, k != 0);
            }
          }
          umma_commit(&sm.acc_full[half]);
        }
        if (alive) umma_commit(&sm.x_empty[stage]);
        if (++stage == XSTAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp < 2 + LN_WARPS) {
    // ---- layer norm, two threads per pair of the tile (lanes l and l ^ 16)
    if (threadIdx.x < 192) (threadIdx.x < 128 ? sm.gamma2 : sm.beta2)[threadIdx.x & 63] = ln_param.word();
    named_barrier(1 + EPI_WARPS / 4, LN_WARPS * 32);
    const int r = (warp - 2) * 16 + (lane & 15);
    int stage = 0;
    uint32_t phase = 0, it = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x, ++it) {
      int o, t;
      locate(tile, o, t);
      t += r;
      float mval = 0.f;
      if (t < p.n_inner) mval = p.mask ? p.mask[o * p.ms_outer + t * p.ms_inner] : 1.0f;
      if (!mbar_wait(&sm.x_full[stage], phase, p.status, ST_TIMEOUT_PROLOGUE)) break;
      __syncwarp();
      ln_row_two_threads(sm.x[stage], r, lane >> 4, sm.gamma2, sm.beta2, p.eps);
      if (lane < 16) sm.mask[it & (MASK_SLOTS - 1)][r] = __float2bfloat16_rn(mval);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.xn_full[stage]);
      if (++stage == XSTAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else {
    // ---- epilogue: thread = output channel (TMEM lane), columns = pairs, 32 per warpgroup
    const int quarter = warp & 3, part = (warp - 2 - LN_WARPS) >> 2;
    const int chan = quarter * 32 + lane;
    const bool leader = quarter == 0 && lane == 0;  // issues the warpgroup's stores
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + part * 32;
    uint8_t* out = sm.out[part];
    uint32_t it = 0;
    bool alive = true;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles && alive; tile += gridDim.x, ++it) {
      int o, t0;
      locate(tile, o, t0);
      t0 += part * 32;
      const uint32_t* mrow = reinterpret_cast<const uint32_t*>(sm.mask[it & (MASK_SLOTS - 1)]) + part * 16;
      for (int half = 0; half < 2; ++half) {
        // the previous tile must have left the staging buffer; the vote makes the outcome of the
        // bounded wait the same for all 128 threads, which meet at a barrier below
        if (leader) tma_store_wait_read();
        if (!named_barrier_and(1 + part, 128, mbar_wait(&sm.acc_full[half], it & 1, p.status, ST_TIMEOUT_EPILOGUE))) {
          alive = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int chunk = 0; chunk < 2; ++chunk) {
          uint32_t pr[16], gr[16];
          tmem_ld16(lane_addr + half * 256 + chunk * 16, pr);
          tmem_ld16(lane_addr + half * 256 + 128 + chunk * 16, gr);
          tmem_ld_wait();
          // bf16 rounding after the two products, the sigmoid, the gating and the
          // mask, as on the reference's bf16 trunk.
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const uint4 m = *reinterpret_cast<const uint4*>(mrow + chunk * 8 + 4 * q);
            const uint32_t mm[4] = {m.x, m.y, m.z, m.w};
            uint32_t packed[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int c = 8 * q + 2 * e;
              const uint32_t pv = pack_bf16x2(__uint_as_float(pr[c]), __uint_as_float(pr[c + 1]));
              const uint32_t sg = sigmoid_bf16x2(__uint_as_float(gr[c]), __uint_as_float(gr[c + 1]));
              packed[e] = bf16x2_mul(bf16x2_mul(sg, pv), mm[e]);
            }
            *reinterpret_cast<uint4*>(out + chan * 64 + (((chunk * 2 + q) ^ ((chan >> 1) & 3)) << 4)) =
                make_uint4(packed[0], packed[1], packed[2], packed[3]);
          }
        }
        tc_fence_before();
        fence_proxy_async();
        named_barrier(1 + part, 128);
        const int whole = RAGGED ? p.n_inner & ~7 : p.n_inner;
        if (leader && t0 < whole) {  // pairs past the tensor's end are not written
          const int block = o / p.rows_per_block;
          tma_store_4d(half ? &tm_b : &tm_a, out, t0, o - block * p.rows_per_block, 0, block);
          tma_store_commit();
        }
        if constexpr (RAGGED) {
          if (t0 <= whole && whole < t0 + 32) {  // (this thread's own row of the staged tile)
            const int block = o / p.rows_per_block;
            __nv_bfloat16* dst = (half ? p.b : p.a) + block * p.block_stride + chan * p.chan_stride +
                                 (o - block * p.rows_per_block) * p.ld + whole;
            const __nv_bfloat16* src =
                reinterpret_cast<const __nv_bfloat16*>(out + chan * 64 + ((((whole - t0) >> 3) ^ ((chan >> 1) & 3)) << 4));
            for (int e = 0; e < p.n_inner - whole; ++e) dst[e] = src[e];
          }
        }
        if (lane == 0) mbar_arrive(&sm.acc_empty[half]);
      }
    }
    status = stores_read_and_status(leader, p.status);
  }

  settle(status, p.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace

}  // namespace b200

extern "C" size_t b200tri_trimul_project_workspace_bytes(void) {
  return 512 * 128 * 2 + 1024;  // copies of weights that are not 16-byte aligned
}

extern "C" int b200tri_trimul_project(const b200tri_trimul_project_args* a, b200tri_stream_t stream) {
  return b200::mul_project_launch(a, false, reinterpret_cast<cudaStream_t>(stream));
}

int b200::mul_project_launch(const b200tri_trimul_project_args* a, bool pad_is_scratch, cudaStream_t stream) {
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "project: null args");
  B200_REQUIRE(a->x && a->a && a->b && a->p_in && a->g_in && a->norm_in_scale && a->norm_in_bias, B200TRI_ERR_INVALID,
               "project: null pointer argument");
  B200_REQUIRE(a->n_outer > 0 && a->n_inner > 0, B200TRI_ERR_INVALID, "project: sizes must be positive");
  B200_REQUIRE(a->xs_outer % 8 == 0 && a->xs_inner % 8 == 0, B200TRI_ERR_INVALID,
               "project: x strides must be multiples of 8 elements");
  B200_REQUIRE(a->ld % 8 == 0 && a->chan_stride % 8 == 0 && a->block_stride % 8 == 0 && a->rows_per_block > 0,
               B200TRI_ERR_INVALID, "project: output pitch/strides must be multiples of 8 elements");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(a->a) | reinterpret_cast<uintptr_t>(a->b)) & 15) == 0, B200TRI_ERR_INVALID,
               "project: outputs must be 16-byte aligned");
  B200_REQUIRE(a->workspace && a->workspace_bytes >= b200tri_trimul_project_workspace_bytes(), B200TRI_ERR_WORKSPACE,
               "project: workspace of %zu bytes needed", b200tri_trimul_project_workspace_bytes());
  int* status = device_status_word();
  B200_REQUIRE(status != nullptr, B200TRI_ERR_CUDA, "project: no current CUDA device");

  // the weights are read in place; the workspace is only for one that is not 16-byte aligned
  const bool chained = pdl_chained();
  Carver ws(a->workspace);
  const void *w_p, *w_g;
  {
    void* s0 = ws.take<__nv_bfloat16>(128 * 256);
    void* s1 = ws.take<__nv_bfloat16>(128 * 256);
    int rc = aligned_weight(a->p_in, 128 * 256 * 2, s0, stream, &w_p);
    if (rc || (rc = aligned_weight(a->g_in, 128 * 256 * 2, s1, stream, &w_g))) return rc;
  }
  CUtensorMap tm_x, tm_p, tm_g;
  {
    const uint64_t dims[3] = {128, (uint64_t)a->n_inner, (uint64_t)a->n_outer};
    const uint64_t str[2] = {(uint64_t)a->xs_inner * 2, (uint64_t)a->xs_outer * 2};
    const uint32_t box[3] = {64, 128, 1};
    int rc = make_tmap(&tm_x, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    int rc = make_weight_map(&tm_p, w_p, 128, 256, 128);
    if (rc || (rc = make_weight_map(&tm_g, w_g, 128, 256, 128))) return rc;
  }
  CUtensorMap tm_out[2];  // (pair, row in block, channel, block), written as tiles of [128 channels][32 pairs]
  const bool ragged = !pad_is_scratch && a->n_inner % 8 != 0;
  const int whole = a->n_inner < 8 ? 8 : a->n_inner & ~7;
  const int rpb = a->rows_per_block < a->n_outer ? a->rows_per_block : a->n_outer;
  for (int i = 0; i < 2; ++i) {
    const int blocks = (a->n_outer + rpb - 1) / rpb;
    const uint64_t dims[4] = {(uint64_t)(ragged ? whole : a->n_inner), (uint64_t)rpb, 128, (uint64_t)blocks};
    const uint64_t str[3] = {(uint64_t)a->ld * 2, (uint64_t)a->chan_stride * 2,
                             (uint64_t)(blocks > 1 ? a->block_stride : a->chan_stride * 128) * 2};
    const uint32_t box[4] = {32, 1, 128, 1};
    int rc = make_tmap(&tm_out[i], i ? a->b : a->a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, dims, str, box, Swz::B64);
    if (rc) return rc;
  }
  RaggedParams p;
  p.n_outer = a->n_outer;
  p.n_inner = a->n_inner;
  p.tiles_inner = (a->n_inner + 127) / 128;
  const long long tiles = static_cast<long long>(p.tiles_inner) * a->n_outer;
  B200_REQUIRE(tiles < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "project: too many tiles (%lld)", tiles);
  p.total_tiles = static_cast<uint32_t>(tiles);
  p.mask = a->mask;
  p.ms_outer = a->ms_outer;
  p.ms_inner = a->ms_inner;
  p.gamma = a->norm_in_scale;
  p.beta = a->norm_in_bias;
  p.early_weights = chained && w_p == a->p_in && w_g == a->g_in;
  p.rows_per_block = rpb;
  p.a = static_cast<__nv_bfloat16*>(a->a);
  p.b = static_cast<__nv_bfloat16*>(a->b);
  p.ld = a->ld;
  p.chan_stride = a->chan_stride;
  p.block_stride = a->block_stride;
  p.eps = a->eps;
  p.status = status;

  const long long grid = tiles < sm_count() ? tiles : sm_count();
  auto go = [&](auto kernel, const auto& params) {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), (int)sizeof(Smem));
    if (rc) return rc;
    TimedLaunch timed(K_TRIMUL_PROJECT, stream);
    return launch(kernel, dim3(static_cast<unsigned>(grid)), dim3(THREADS), sizeof(Smem), stream, true, tm_x, tm_p, tm_g,
                  tm_out[0], tm_out[1], params);
  };
  return ragged ? go(project_kernel<true>, p) : go(project_kernel<false>, static_cast<const ProjParams&>(p));
}
