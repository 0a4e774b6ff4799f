// Triangle multiplicative update, output stage.
//
//   out[i][j][:] = LN_out(t[:, i, j]) @ p_out * sigmoid(LN_in(x[i][j]) @ g_out)  (+ residual)
//
// Reference: src/foldjax/models/boltz2/models/triangle/triangle.py:124-129.
// t is the contraction result, channel-major (t[d][i][j]); the kernel turns it
// back into channel-last while it normalises. The output gate is recomputed
// from x here instead of being stored by the projection stage: reading x costs
// the same bytes as reading a stored gate would, and saves writing it.
//
// One tile = 128 consecutive pairs (i, j0..j0+127). Persistent, one CTA per SM:
//   warp 0       TMA producer: two 128x128 weights once; per tile the x tile
//                (K-major, swizzled) and the t tile ([channel][pair], two swizzled slabs of 64 pairs)
//   warp 1       MMA issuer: D1 = LN_in(x) . g_out^T, D2 = LN_out(t) . p_out^T
//                (warps 2 and 3 idle: registers move between whole warpgroups)
//   warps 4-7    layer norm of x in place, one thread per pair
//   warps 8-11   layer norm of t, one thread per pair: the tile is turned into operand layout in
//                place (read column, mbarrier, write row), which holds a row in registers
//   warps 12-19  epilogue: D2 * sigmoid(D1) (+ residual) -> bf16 -> shared-memory tile -> TMA
//                store, 64 channels per warpgroup, the residual fetched before the products are
//                waited for
// TMEM: 2 x (D1, D2) so the epilogue overlaps the next tile's MMAs.
//
// Bound: HBM (read t and x, write out: 3 * n_i*n_j*128*2 bytes; + residual) by the bytes; in fact
// the layer norms, chains of 192 dependent additions per row beside 900 other instructions: the warps of x are
// at it 97 % of the time (t 68 %, epilogue 77 %), at five warps per scheduler. n = 1024: 247 us with one
// warpgroup for both layer norms and one thread per row of the residual, 226 with two (123 by the bytes); by events
// around the launch at n = 1003 258 with four words of x at a time and a store per warpgroup, 248 with eight
// and a store per warp. Measured and not better: x in registers (spills), two threads per row whose
// chains follow each other (263), alternate warpgroups per tile, t transposed by ldmatrix.
#include "host.cuh"
#include "ln.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int STAGES = 2;
constexpr int TILE_BYTES = 2 * SLAB_BYTES;
constexpr int WORK_WARPS = 8, EPI_WARPS = 8;  // half of the working warps per layer norm
constexpr int THREADS = 128 + (WORK_WARPS + EPI_WARPS) * 32;

struct Smem {
  uint8_t w[4 * SLAB_BYTES];  // g_out, p_out: two boxes [128 in][64 out] each, MN-major
  uint8_t x[STAGES][TILE_BYTES];
  uint8_t t[STAGES][TILE_BYTES];
  uint8_t out[TILE_BYTES];  // two slabs of 64 channels, one per epilogue warpgroup
  alignas(16) uint32_t gamma_in[64], beta_in[64], gamma_out[64], beta_out[64];
  uint64_t w_full, in_full[STAGES], xn_full[STAGES], in_empty[STAGES], col_read[STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_base;
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

struct FinishParams {
  int n_i, n_j, tiles_j;
  uint32_t total_tiles;
  const void* ln[4];    // gamma_in, beta_in, gamma_out, beta_out
  bool early_weights;   // the weights may be read before pdl_wait()
  const __nv_bfloat16* residual;
  long long os_i, os_j;
  float eps;
  int t_rpb;  // rows per block of t
  int* status;
};

__global__ void __launch_bounds__(THREADS, 1)
finish_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_t,
              const __grid_constant__ CUtensorMap tm_g, const __grid_constant__ CUtensorMap tm_p,
              const __grid_constant__ CUtensorMap tm_out, const FinishParams p) {
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
    tma_prefetch_desc(&tm_t);
    tma_prefetch_desc(&tm_g);
    tma_prefetch_desc(&tm_p);
    mbar_init(&sm.w_full, 1);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sm.in_full[s], 1);
      mbar_init(&sm.xn_full[s], WORK_WARPS);
      mbar_init(&sm.in_empty[s], 1);
      mbar_init(&sm.col_read[s], WORK_WARPS / 2);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sm.acc_full[a], 1);
      mbar_init(&sm.acc_empty[a], EPI_WARPS);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  if (!p.early_weights) pdl_wait();
  LnParam ln_param;
  if (threadIdx.x >= 128 && threadIdx.x < 384)
    ln_param.request(threadIdx.x < 192   ? p.ln[0]
                     : threadIdx.x < 256 ? p.ln[1]
                     : threadIdx.x < 320 ? p.ln[2]
                                         : p.ln[3],
                     threadIdx.x & 63);
  if (warp == 0 && lane == 0) {  // (the thread that initialised the barrier)
    mbar_expect_tx(&sm.w_full, 4 * SLAB_BYTES);
    for (int g = 0; g < 2; ++g)
      for (int s = 0; s < 2; ++s)
        tma_load_2d(sm.w + (g * 2 + s) * SLAB_BYTES, g ? &tm_p : &tm_g, &sm.w_full, s * 64, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;
  int status = -1;

  // (32-bit: a 64-bit division costs a role hundreds of cycles per tile)
  auto locate = [&](uint32_t tile, int& i, int& j0) {
    const uint32_t q = tile / static_cast<uint32_t>(p.tiles_j);
    i = q;
    j0 = (tile - q * p.tiles_j) * 128;
  };
  auto load_in = [&](int stage, int i, int j0, int block, int in_block) {
    mbar_expect_tx(&sm.in_full[stage], 2 * TILE_BYTES);
    tma_load_3d(sm.x[stage], &tm_x, &sm.in_full[stage], 0, j0, i);
    tma_load_3d(sm.x[stage] + SLAB_BYTES, &tm_x, &sm.in_full[stage], 64, j0, i);
    for (int half = 0; half < 2; ++half)
      tma_load_4d(sm.t[stage] + half * SLAB_BYTES, &tm_t, &sm.in_full[stage], j0 + half * 64, in_block, 0, block);
  };
  int first_i, first_j0;  // the first tile, located ahead of the wait and requested right behind it
  locate(blockIdx.x, first_i, first_j0);
  const int first_block = first_i / p.t_rpb;
  if (p.early_weights) pdl_wait();
  if (threadIdx.x == 0) load_in(0, first_i, first_j0, first_block, first_i - first_block * p.t_rpb);
  pdl_trigger();

  // 640 threads x 96 registers = 128 x (40 + 88 + 144 + 2 x 104)
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
      if (elect_one()) {
        int stage = 1;  // (stage 0 has the first tile)
        uint32_t phase = 0;
        for (uint32_t tile = blockIdx.x + gridDim.x; tile < p.total_tiles; tile += gridDim.x) {
          int i, j0;
          locate(tile, i, j0);
          const int block = i / p.t_rpb;
          if (!mbar_wait(&sm.in_empty[stage], phase ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
          load_in(stage, i, j0, block, i - block * p.t_rpb);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    } else if (warp == 1) {
      if (elect_one()) {
        constexpr uint32_t idesc = umma_idesc_bf16(128, 128) | UMMA_B_MN;
        bool alive = mbar_wait(&sm.w_full, 0, p.status, ST_TIMEOUT_MMA);
        int stage = 0;
        uint32_t phase = 0, it = 0;
        for (uint32_t tile = blockIdx.x; tile < p.total_tiles && alive; tile += gridDim.x, ++it) {
          const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
          if (!mbar_wait(&sm.acc_empty[acc], acc_phase ^ 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.xn_full[stage], phase, p.status, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const uint32_t d_tmem = tmem_base + acc * 256 + g * 128;
            const uint32_t in = smem_u32(g == 0 ? sm.x[stage] : sm.t[stage]);
            const uint64_t bdesc = umma_desc_mnmajor(smem_u32(sm.w + g * 2 * SLAB_BYTES), SLAB_BYTES);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const uint64_t adesc = umma_desc_kmajor(in + (k >> 2) * SLAB_BYTES, 128);
              umma_bf16_ss(d_tmem, umma_desc_advance(adesc, (k & 3) * 32), umma_desc_advance(bdesc, k * 2048), idesc, k != 0);
            }
          }
          umma_commit(&sm.in_empty[stage]);
          umma_commit(&sm.acc_full[acc]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp < 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    (threadIdx.x < 192 ? sm.gamma_in : sm.beta_in)[threadIdx.x & 63] = ln_param.word();
    named_barrier(1, 128);
    const int r = threadIdx.x - 128;  // pair of the tile
    int stage = 0;
    uint32_t phase = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x) {
      if (!mbar_wait(&sm.in_full[stage], phase, p.status, ST_TIMEOUT_PROLOGUE)) break;
      ln_row_sweeps<8>(sm.x[stage], r, sm.gamma_in, sm.beta_in, p.eps);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.xn_full[stage]);
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else if (warp < 12) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    (threadIdx.x < 320 ? sm.gamma_out : sm.beta_out)[threadIdx.x & 63] = ln_param.word();
    named_barrier(2, 128);
    const int r = threadIdx.x - 256;  // pair of the tile
    int stage = 0;
    uint32_t phase = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x) {
      if (!mbar_wait(&sm.in_full[stage], phase, p.status, ST_TIMEOUT_PROLOGUE)) break;
      uint4 v[16];
      {
        const uint8_t* slab = sm.t[stage] + (r >> 6) * SLAB_BYTES;
        uint32_t* w = reinterpret_cast<uint32_t*>(v);
#pragma unroll
        for (int i = 0; i < 64; ++i) {  // channels 2 * i and 2 * i + 1 of this pair
          const uint32_t lo = *reinterpret_cast<const unsigned short*>(slab + sw128_offset(2 * i, (r & 63) >> 3) + (r & 7) * 2);
          const uint32_t hi = *reinterpret_cast<const unsigned short*>(slab + sw128_offset(2 * i + 1, (r & 63) >> 3) + (r & 7) * 2);
          w[i] = lo | (hi << 16);
        }
        // Rows may overwrite the tile only once every column has been read.
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.col_read[stage]);
        ln_row_words(v, sm.gamma_out, sm.beta_out, p.eps);
        if (!mbar_wait(&sm.col_read[stage], phase, p.status, ST_TIMEOUT_PROLOGUE)) break;
        ln_store_row(sm.t[stage], r, v);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.xn_full[stage]);
      if (++stage == STAGES) {
        stage = 0;
        phase ^= 1;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int quarter = warp & 3, half = (warp - 12) >> 2;  // 64 channels per warpgroup
    const int pr = quarter * 32 + lane;  // pair inside the tile = TMEM lane
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * 64;
    uint8_t* stage_out = sm.out + half * SLAB_BYTES;
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x, ++it) {
      int i, j0;
      locate(tile, i, j0);
      const uint32_t acc = it & 1, acc_phase = (it >> 1) & 1;
      uint4 res[8];  // residual of the warp's 32 pairs, 8 lanes to a pair's 64 channels (whole lines)
      if (p.residual) {
        const int t = j0 + quarter * 32 + (lane >> 3);
        const __nv_bfloat16* src = p.residual + static_cast<long long>(i) * p.os_i + half * 64 + (lane & 7) * 8;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          res[q] = t + 4 * q < p.n_j ? *reinterpret_cast<const uint4*>(src + static_cast<long long>(t + 4 * q) * p.os_j)
                                      : make_uint4(0u, 0u, 0u, 0u);
      }
      // (a vote: TMEM accesses take the whole warp. Each warp stages and stores its own 32 pairs)
      if (!__all_sync(0xffffffffu, mbar_wait(&sm.acc_full[acc], acc_phase, p.status, ST_TIMEOUT_EPILOGUE))) break;
      tc_fence_after();
      if (lane == 0) tma_store_wait_read();  // the previous tile has left them
      __syncwarp();
#pragma unroll 1  // (the roles' unrolled code competes for the instruction cache)
      for (int chunk = 0; chunk < 4; ++chunk) {
        uint32_t g[16], o[16];
        tmem_ld16(lane_addr + acc * 256 + chunk * 16, g);
        tmem_ld16(lane_addr + acc * 256 + 128 + chunk * 16, o);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t u[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = 8 * q + 2 * e;
            const uint32_t ov = pack_bf16x2(__uint_as_float(o[c]), __uint_as_float(o[c + 1]));
            const uint32_t sg = sigmoid_bf16x2(__uint_as_float(g[c]), __uint_as_float(g[c + 1]));
            u[e] = bf16x2_mul(ov, sg);
          }
          *reinterpret_cast<uint4*>(stage_out + sw128_offset(pr, chunk * 2 + q)) = make_uint4(u[0], u[1], u[2], u[3]);
        }
      }
      if (p.residual) {  // the caller's z + update, one more bf16 rounding, in the residual's arrangement
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          uint4* ptr = reinterpret_cast<uint4*>(stage_out + sw128_offset(quarter * 32 + 4 * q + (lane >> 3), lane & 7));
          uint4 u = *ptr;
          u.x = bf16x2_add(res[q].x, u.x);
          u.y = bf16x2_add(res[q].y, u.y);
          u.z = bf16x2_add(res[q].z, u.z);
          u.w = bf16x2_add(res[q].w, u.w);
          *ptr = u;
        }
      }
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0 && j0 + quarter * 32 < p.n_j) {  // rows past n_j are outside the tensor and are not written
        tma_store_3d(&tm_out, stage_out + quarter * 4096, half * 64, j0 + quarter * 32, i);
        tma_store_commit();
      }
      if (lane == 0) mbar_arrive(&sm.acc_empty[acc]);
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

extern "C" size_t b200tri_trimul_finish_workspace_bytes(void) { return 256 * 128 * 2 + 1024 + 1024; }

extern "C" int b200tri_trimul_finish(const b200tri_trimul_finish_args* a, b200tri_stream_t stream_) {
  using namespace b200;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "finish: null args");
  B200_REQUIRE(a->t && a->x && a->out && a->p_out && a->g_out && a->norm_in_scale && a->norm_in_bias &&
                   a->norm_out_scale && a->norm_out_bias,
               B200TRI_ERR_INVALID, "finish: null pointer argument");
  B200_REQUIRE(a->n_i > 0 && a->n_j > 0, B200TRI_ERR_INVALID, "finish: sizes must be positive");
  B200_REQUIRE(a->t_ld % 8 == 0 && a->t_chan_stride % 8 == 0 && a->xs_i % 8 == 0 && a->xs_j % 8 == 0 &&
                   a->os_i % 8 == 0 && a->os_j % 8 == 0,
               B200TRI_ERR_INVALID, "finish: pitches and strides must be multiples of 8 elements");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(a->out) | reinterpret_cast<uintptr_t>(a->residual)) & 15) == 0,
               B200TRI_ERR_INVALID, "finish: out/residual must be 16-byte aligned");
  B200_REQUIRE(a->workspace && a->workspace_bytes >= b200tri_trimul_finish_workspace_bytes(), B200TRI_ERR_WORKSPACE,
               "finish: workspace of %zu bytes needed", b200tri_trimul_finish_workspace_bytes());
  int* status = device_status_word();
  B200_REQUIRE(status != nullptr, B200TRI_ERR_CUDA, "finish: no current CUDA device");

  // the weights are read in place; the workspace is only for one that is not 16-byte aligned
  Carver ws(a->workspace);
  const void *w_g, *w_p;
  {
    void* s0 = ws.take<__nv_bfloat16>(128 * 128);
    void* s1 = ws.take<__nv_bfloat16>(128 * 128);
    int rc = aligned_weight(a->g_out, 128 * 128 * 2, s0, stream, &w_g);
    if (rc || (rc = aligned_weight(a->p_out, 128 * 128 * 2, s1, stream, &w_p))) return rc;
  }
  CUtensorMap tm_x, tm_t, tm_g, tm_p, tm_out;
  {
    const uint64_t dims[3] = {128, (uint64_t)a->n_j, (uint64_t)a->n_i};
    const uint64_t str[2] = {(uint64_t)a->os_j * 2, (uint64_t)a->os_i * 2};
    const uint32_t box[3] = {64, 32, 1};
    int rc = make_tmap(&tm_out, a->out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    const uint64_t dims[3] = {128, (uint64_t)a->n_j, (uint64_t)a->n_i};
    const uint64_t str[2] = {(uint64_t)a->xs_j * 2, (uint64_t)a->xs_i * 2};
    const uint32_t box[3] = {64, 128, 1};
    int rc = make_tmap(&tm_x, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    // (j, row in block, channel, block); one block when t is not row-blocked
    const bool blocked = a->t_rows_per_block > 0 && a->t_rows_per_block < a->n_i;
    const uint64_t rpb = blocked ? (uint64_t)a->t_rows_per_block : (uint64_t)a->n_i;
    const uint64_t blocks = (a->n_i + rpb - 1) / rpb;
    B200_REQUIRE(!blocked || a->t_block_stride % 8 == 0, B200TRI_ERR_INVALID, "finish: t_block_stride must be a multiple of 8");
    const uint64_t dims[4] = {(uint64_t)a->n_j, rpb, 128, blocks};
    const uint64_t str[3] = {(uint64_t)a->t_ld * 2, (uint64_t)a->t_chan_stride * 2,
                             (uint64_t)(blocked ? a->t_block_stride : a->t_chan_stride * 128) * 2};
    const uint32_t box[4] = {64, 1, 128, 1};
    int rc = make_tmap(&tm_t, a->t, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    int rc = make_weight_map(&tm_g, w_g, 128, 128, 128);
    if (rc || (rc = make_weight_map(&tm_p, w_p, 128, 128, 128))) return rc;
  }
  FinishParams p;
  p.n_i = a->n_i;
  p.n_j = a->n_j;
  p.tiles_j = (a->n_j + 127) / 128;
  const long long tiles = static_cast<long long>(p.tiles_j) * a->n_i;
  B200_REQUIRE(tiles < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "finish: too many tiles (%lld)", tiles);
  p.total_tiles = static_cast<uint32_t>(tiles);
  p.ln[0] = a->norm_in_scale;
  p.ln[1] = a->norm_in_bias;
  p.ln[2] = a->norm_out_scale;
  p.ln[3] = a->norm_out_bias;
  p.early_weights = pdl_chained() && w_g == a->g_out && w_p == a->p_out;
  p.residual = static_cast<const __nv_bfloat16*>(a->residual);
  p.os_i = a->os_i;
  p.os_j = a->os_j;
  p.eps = a->eps;
  p.t_rpb = (a->t_rows_per_block > 0 && a->t_rows_per_block < a->n_i) ? a->t_rows_per_block : a->n_i;
  p.status = status;

  {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(finish_kernel), (int)sizeof(Smem));
    if (rc) return rc;
  }
  const long long grid = tiles < sm_count() ? tiles : sm_count();
  {
    TimedLaunch timed(K_TRIMUL_FINISH, stream);
    return launch(finish_kernel, dim3(static_cast<unsigned>(grid)), dim3(THREADS), sizeof(Smem), stream, true, tm_x, tm_t,
                  tm_g, tm_p, tm_out, p);
  }
}
