// Triangle attention, output stage.
//
//   g    = bf16(sigmoid(bf16(LN(x) @ Wg)))
//   out  = bf16(bf16(o * g) @ Wo)   (+ residual), written through caller strides so the
//          ending node lands transposed back in place
//
// Reference: src/foldjax/models/boltz2/models/triangle/triangle_attention.py
// :360-366 (gate projection), :421-425 (gating, output projection), :160-161.
// o is the attention core's output [n_outer][n_inner][128] in the attention
// frame; x and out are addressed as base + o*stride_outer + t*stride_inner.
//
// One tile = 128 consecutive pairs. Persistent, one CTA per SM:
//   warp 0       TMA producer (Wg, Wo once; x tiles in a 2-stage ring, o tiles in a 3-stage ring)
//   warp 1       MMA issuer: G = LN(x).Wg^T, then OUT = (o*g).Wo^T
//                (warps 2 and 3 idle: registers move between whole warpgroups)
//   warps 4-7    layer norm of x in place, one thread per pair, the row in its registers
//   warps 8-11   gating of o in place, one thread per pair (the o tile becomes the A operand of the
//                second product)
//   warps 12-15  epilogue of OUT: residual fetched before the product is waited for, sum staged in
//                the o tile (dead by then), TMA stores per warp
// Bound: HBM (read x and o, write out: 3 * n*n*128*2 bytes; + residual) - once enough warps
// hide the latencies of TMEM and of the row-wise accesses.
#include "host.cuh"
#include "ln.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int XSTAGES = 2, OSTAGES = 3;  // an x tile is free after the first product, an o tile once it is stored
constexpr int TILE_BYTES = 2 * SLAB_BYTES;
constexpr int LN_WARPS = 4, GATE_WARPS = 4, EPI_WARPS = 4;
constexpr int THREADS = 128 + (LN_WARPS + GATE_WARPS + EPI_WARPS) * 32;

struct Smem {
  uint8_t w[4 * SLAB_BYTES];  // Wg, Wo: two boxes [128 in][64 out] each, MN-major
  uint8_t x[XSTAGES][TILE_BYTES];
  uint8_t o[OSTAGES][TILE_BYTES];
  alignas(16) uint32_t gamma2[64], beta2[64];
  uint64_t w_full, x_full[XSTAGES], xn_full[XSTAGES], x_empty[XSTAGES], o_full[OSTAGES], y_full[OSTAGES], o_empty[OSTAGES];
  uint64_t g_full[2], g_empty[2], out_full[2], out_empty[2];
  uint32_t tmem_base;
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

struct Params {
  int n_outer, n_inner, tiles_inner;
  uint32_t total_tiles;
  const void* gamma;
  const void* beta;
  bool early_weights;  // the weights may be read before pdl_wait()
  const __nv_bfloat16* residual;
  long long os_outer, os_inner;
  float eps;
  int* status;
};

__global__ void __launch_bounds__(THREADS, 1)
att_finish_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_o,
                  const __grid_constant__ CUtensorMap tm_wg, const __grid_constant__ CUtensorMap tm_wo,
                  const __grid_constant__ CUtensorMap tm_out, const Params p) {
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
    tma_prefetch_desc(&tm_o);
    tma_prefetch_desc(&tm_wg);
    tma_prefetch_desc(&tm_wo);
    mbar_init(&sm.w_full, 1);
    for (int s = 0; s < XSTAGES; ++s) {
      mbar_init(&sm.x_full[s], 1);
      mbar_init(&sm.xn_full[s], LN_WARPS);
      mbar_init(&sm.x_empty[s], 1);
    }
    for (int s = 0; s < OSTAGES; ++s) {
      mbar_init(&sm.o_full[s], 1);
      mbar_init(&sm.y_full[s], GATE_WARPS);
      mbar_init(&sm.o_empty[s], EPI_WARPS);  // their stores
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sm.g_full[a], 1);
      mbar_init(&sm.g_empty[a], GATE_WARPS);
      mbar_init(&sm.out_full[a], 1);
      mbar_init(&sm.out_empty[a], EPI_WARPS);
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
  if (warp == 0 && lane == 0) {  // (the thread that initialised the barrier)
    mbar_expect_tx(&sm.w_full, 4 * SLAB_BYTES);
    for (int g = 0; g < 2; ++g)
      for (int s = 0; s < 2; ++s)
        tma_load_2d(sm.w + (g * 2 + s) * SLAB_BYTES, g ? &tm_wo : &tm_wg, &sm.w_full, s * 64, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;
  // TMEM: buffer a (= tile parity): G at a*256, OUT at a*256 + 128.
  int status = -1;

  // (32-bit: a 64-bit division costs a role hundreds of cycles per tile)
  auto locate = [&](uint32_t tile, int& o, int& t0) {
    const uint32_t q = tile / static_cast<uint32_t>(p.tiles_inner);
    o = q;
    t0 = (tile - q * p.tiles_inner) * 128;
  };
  auto load_x = [&](int xs, int o, int t0) {
    mbar_expect_tx(&sm.x_full[xs], TILE_BYTES);
    tma_load_3d(sm.x[xs], &tm_x, &sm.x_full[xs], 0, t0, o);
    tma_load_3d(sm.x[xs] + SLAB_BYTES, &tm_x, &sm.x_full[xs], 64, t0, o);
  };
  auto load_o = [&](int os, int o, int t0) {
    mbar_expect_tx(&sm.o_full[os], TILE_BYTES);
    tma_load_3d(sm.o[os], &tm_o, &sm.o_full[os], 0, t0, o);
    tma_load_3d(sm.o[os] + SLAB_BYTES, &tm_o, &sm.o_full[os], 64, t0, o);
  };
  int first_o, first_t0;  // the first tile, located ahead of the wait and requested right behind it
  locate(blockIdx.x, first_o, first_t0);
  if (p.early_weights) pdl_wait();
  if (threadIdx.x == 0) {
    load_x(0, first_o, first_t0);
    load_o(0, first_o, first_t0);
  }
  pdl_trigger();
  const uint32_t n_my = blockIdx.x < p.total_tiles ? (p.total_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

  // 512 threads x 128 registers = 128 x (72 + 144 + 128 + 168)
  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  if (warp == 0) {
    if (elect_one()) {
      uint32_t it = 1;  // (the first tile is on its way)
      for (uint32_t tile = blockIdx.x + gridDim.x; tile < p.total_tiles; tile += gridDim.x, ++it) {
        int o, t0;
        locate(tile, o, t0);
        const uint32_t xs = it % XSTAGES, os = it % OSTAGES;
        if (!mbar_wait(&sm.x_empty[xs], ((it / XSTAGES) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
        load_x(xs, o, t0);
        if (!mbar_wait(&sm.o_empty[os], ((it / OSTAGES) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
        load_o(os, o, t0);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 128) | UMMA_B_MN;
      bool alive = mbar_wait(&sm.w_full, 0, p.status, ST_TIMEOUT_MMA);
      // Two products per tile; the second of tile t is issued after the first of
      // tile t+1, mirroring the order in which the gating warps deliver operands.
      auto product = [&](uint32_t d_tmem, uint32_t a_smem, int wgroup) {
        const uint64_t bdesc = umma_desc_mnmajor(smem_u32(sm.w + wgroup * 2 * SLAB_BYTES), SLAB_BYTES);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint64_t adesc = umma_desc_kmajor(a_smem + (k >> 2) * SLAB_BYTES, 128);
          umma_bf16_ss(d_tmem, umma_desc_advance(adesc, (k & 3) * 32), umma_desc_advance(bdesc, k * 2048), idesc, k != 0);
        }
      };
      for (uint32_t it = 0; it <= n_my && alive; ++it) {
        if (it < n_my) {  // first product of tile `it`
          const uint32_t stage = it % XSTAGES, phase = (it / XSTAGES) & 1;
          const uint32_t a = static_cast<uint32_t>(it & 1), aph = static_cast<uint32_t>((it >> 1) & 1);
          if (!mbar_wait(&sm.g_empty[a], aph ^ 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.xn_full[stage], phase, p.status, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
          product(tmem_base + a * 256, smem_u32(sm.x[stage]), 0);
          umma_commit(&sm.x_empty[stage]);
          umma_commit(&sm.g_full[a]);
        }
        if (it > 0) {  // second product of tile `it - 1`
          const uint32_t jt = it - 1;
          const uint32_t stage = jt % OSTAGES, phase = (jt / OSTAGES) & 1;
          const uint32_t a = static_cast<uint32_t>(jt & 1), aph = static_cast<uint32_t>((jt >> 1) & 1);
          if (!mbar_wait(&sm.out_empty[a], aph ^ 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.y_full[stage], phase, p.status, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
          product(tmem_base + a * 256 + 128, smem_u32(sm.o[stage]), 1);
          umma_commit(&sm.out_full[a]);
        }
      }
    }
  } else if (warp >= 4 && warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    const int row = (warp - 4) * 32 + lane;
    for (uint32_t it = 0; it < n_my; ++it) {
      const uint32_t stage = it % XSTAGES, phase = (it / XSTAGES) & 1;
      if (!mbar_wait(&sm.x_full[stage], phase, p.status, ST_TIMEOUT_PROLOGUE)) break;
      uint4 v[16];
      ln_load_row(sm.x[stage], row, v);
      ln_row_words(v, sm.gamma2, sm.beta2, p.eps);
      ln_store_row(sm.x[stage], row, v);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.xn_full[stage]);
    }
  } else if (warp >= 8 && warp < 12) {  // o <- bf16(o * bf16(sigmoid(bf16(G))))
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    for (uint32_t it = 0; it < n_my; ++it) {
      const uint32_t stage = it % OSTAGES, phase = (it / OSTAGES) & 1;
      const uint32_t a = it & 1, aph = (it >> 1) & 1;
      if (!mbar_wait(&sm.o_full[stage], phase, p.status, ST_TIMEOUT_PROLOGUE) ||
          !mbar_wait(&sm.g_full[a], aph, p.status, ST_TIMEOUT_PROLOGUE))
        break;
      __syncwarp();
      tc_fence_after();
#pragma unroll 1
      for (int chunk = 0; chunk < 4; ++chunk) {  // 32 channels = 4 sixteen-byte chunks of one slab
        uint32_t g[32];
        tmem_ld32(lane_addr + a * 256 + chunk * 32, g);
        tmem_ld_wait();
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
          uint4* ptr = reinterpret_cast<uint4*>(sm.o[stage] + (chunk >> 1) * SLAB_BYTES + sw128_offset(row, (chunk & 1) * 4 + c4));
          uint4 ov = *ptr;
          ov.x = bf16x2_mul(ov.x, sigmoid_bf16x2(__uint_as_float(g[8 * c4 + 0]), __uint_as_float(g[8 * c4 + 1])));
          ov.y = bf16x2_mul(ov.y, sigmoid_bf16x2(__uint_as_float(g[8 * c4 + 2]), __uint_as_float(g[8 * c4 + 3])));
          ov.z = bf16x2_mul(ov.z, sigmoid_bf16x2(__uint_as_float(g[8 * c4 + 4]), __uint_as_float(g[8 * c4 + 5])));
          ov.w = bf16x2_mul(ov.w, sigmoid_bf16x2(__uint_as_float(g[8 * c4 + 6]), __uint_as_float(g[8 * c4 + 7])));
          *ptr = ov;
        }
      }
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sm.y_full[stage]);
        mbar_arrive(&sm.g_empty[a]);
      }
    }
  } else if (warp >= 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + 128;
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x, ++it) {
      int o, t0;
      locate(tile, o, t0);
      t0 += quarter * 32;  // the warp's first pair
      const uint32_t a = it & 1, aph = (it >> 1) & 1;
      uint4 res[2][8];  // residual of the warp's 32 pairs, 8 lanes to a pair's 64 channels (whole lines)
      if (p.residual) {
        const int t = t0 + (lane >> 3);
        const __nv_bfloat16* src = p.residual + static_cast<long long>(o) * p.os_outer + (lane & 7) * 8;
#pragma unroll
        for (int q = 0; q < 16; ++q)
          res[q >> 3][q & 7] = t + 4 * (q & 7) < p.n_inner
                                   ? *reinterpret_cast<const uint4*>(src + static_cast<long long>(t + 4 * (q & 7)) * p.os_inner +
                                                                     (q >> 3) * 64)
                                   : make_uint4(0u, 0u, 0u, 0u);
      }
      if (!mbar_wait(&sm.out_full[a], aph, p.status, ST_TIMEOUT_EPILOGUE)) break;
      __syncwarp();
      tc_fence_after();
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // 64 channels at a time
        uint8_t* stage_out = sm.o[it % OSTAGES] + half * SLAB_BYTES;
#pragma unroll
        for (int chunk = 0; chunk < 4; ++chunk) {
          uint32_t v[16];
          tmem_ld16(lane_addr + a * 256 + half * 64 + chunk * 16, v);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t u[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              u[e] = pack_bf16x2(__uint_as_float(v[8 * q + 2 * e]), __uint_as_float(v[8 * q + 2 * e + 1]));
            *reinterpret_cast<uint4*>(stage_out + sw128_offset(row, chunk * 2 + q)) = make_uint4(u[0], u[1], u[2], u[3]);
          }
        }
        if (p.residual) {  // the caller's z + update, one more bf16 rounding, in the residual's arrangement
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            uint4* ptr = reinterpret_cast<uint4*>(stage_out + sw128_offset(quarter * 32 + 4 * q + (lane >> 3), lane & 7));
            uint4 u = *ptr;
            u.x = bf16x2_add(res[half][q].x, u.x);
            u.y = bf16x2_add(res[half][q].y, u.y);
            u.z = bf16x2_add(res[half][q].z, u.z);
            u.w = bf16x2_add(res[half][q].w, u.w);
            *ptr = u;
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && t0 < p.n_inner) {  // rows past n_inner are outside the tensor and are not written
          tma_store_3d(&tm_out, stage_out + quarter * 4096, half * 64, t0, o);
          tma_store_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sm.out_empty[a]);
        tma_store_wait_read();
        mbar_arrive(&sm.o_empty[it % OSTAGES]);
      }
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

extern "C" size_t b200tri_triatt_finish_workspace_bytes(void) { return 256 * 128 * 2 + 1024 + 1024; }

extern "C" int b200tri_triatt_finish(const b200tri_triatt_finish_args* a, b200tri_stream_t stream_) {
  using namespace b200;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "att finish: null args");
  B200_REQUIRE(a->o && a->x && a->out && a->norm_scale && a->norm_bias && a->w_g && a->w_o, B200TRI_ERR_INVALID,
               "att finish: null pointer argument");
  B200_REQUIRE(a->n_outer > 0 && a->n_inner > 0, B200TRI_ERR_INVALID, "att finish: sizes must be positive");
  B200_REQUIRE(a->xs_outer % 8 == 0 && a->xs_inner % 8 == 0 && a->os_outer % 8 == 0 && a->os_inner % 8 == 0,
               B200TRI_ERR_INVALID, "att finish: strides must be multiples of 8 elements");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(a->out) | reinterpret_cast<uintptr_t>(a->residual)) & 15) == 0,
               B200TRI_ERR_INVALID, "att finish: out/residual must be 16-byte aligned");
  B200_REQUIRE(a->workspace && a->workspace_bytes >= b200tri_triatt_finish_workspace_bytes(), B200TRI_ERR_WORKSPACE,
               "att finish: workspace of %zu bytes needed", b200tri_triatt_finish_workspace_bytes());
  int* status = device_status_word();
  B200_REQUIRE(status != nullptr, B200TRI_ERR_CUDA, "att finish: no current CUDA device");

  // the weights are read in place; the workspace is only for one that is not 16-byte aligned
  Carver ws(a->workspace);
  const void *w_g, *w_o;
  {
    void* s0 = ws.take<__nv_bfloat16>(128 * 128);
    void* s1 = ws.take<__nv_bfloat16>(128 * 128);
    int rc = aligned_weight(a->w_g, 128 * 128 * 2, s0, stream, &w_g);
    if (rc || (rc = aligned_weight(a->w_o, 128 * 128 * 2, s1, stream, &w_o))) return rc;
  }
  CUtensorMap tm_x, tm_o, tm_wg, tm_wo, tm_out;
  {  // the result through the caller's strides (the ending node lands transposed back in place)
    const uint64_t dims[3] = {128, (uint64_t)a->n_inner, (uint64_t)a->n_outer};
    const uint64_t str[2] = {(uint64_t)a->os_inner * 2, (uint64_t)a->os_outer * 2};
    const uint32_t box[3] = {64, 32, 1};
    int rc = make_tmap(&tm_out, a->out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    const uint64_t dims[3] = {128, (uint64_t)a->n_inner, (uint64_t)a->n_outer};
    const uint64_t str[2] = {(uint64_t)a->xs_inner * 2, (uint64_t)a->xs_outer * 2};
    const uint32_t box[3] = {64, 128, 1};
    int rc = make_tmap(&tm_x, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    const uint64_t dims[3] = {128, (uint64_t)a->n_inner, (uint64_t)a->n_outer};
    const uint64_t str[2] = {256, (uint64_t)a->n_inner * 256};
    const uint32_t box[3] = {64, 128, 1};
    int rc = make_tmap(&tm_o, a->o, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    int rc = make_weight_map(&tm_wg, w_g, 128, 128, 128);
    if (rc || (rc = make_weight_map(&tm_wo, w_o, 128, 128, 128))) return rc;
  }
  Params p;
  p.n_outer = a->n_outer;
  p.n_inner = a->n_inner;
  p.tiles_inner = (a->n_inner + 127) / 128;
  const long long tiles = static_cast<long long>(p.tiles_inner) * a->n_outer;
  B200_REQUIRE(tiles < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "att finish: too many tiles (%lld)", tiles);
  p.total_tiles = static_cast<uint32_t>(tiles);
  p.gamma = a->norm_scale;
  p.beta = a->norm_bias;
  p.early_weights = pdl_chained() && w_g == a->w_g && w_o == a->w_o;
  p.residual = static_cast<const __nv_bfloat16*>(a->residual);
  p.os_outer = a->os_outer;
  p.os_inner = a->os_inner;
  p.eps = a->eps;
  p.status = status;

  {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(att_finish_kernel), (int)sizeof(Smem));
    if (rc) return rc;
  }
  const long long grid = tiles < sm_count() ? tiles : sm_count();
  {
    TimedLaunch timed(K_TRIATT_FINISH, stream);
    return launch(att_finish_kernel, dim3(static_cast<unsigned>(grid)), dim3(THREADS), sizeof(Smem), stream, true, tm_x, tm_o,
                  tm_wg, tm_wo, tm_out, p);
  }
}
