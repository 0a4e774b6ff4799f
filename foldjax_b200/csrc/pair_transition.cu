// Pair transition (SwiGLU feed-forward on every pair), fused into one pass over z.
//
//   xn     = LN(x)
//   a, b   = bf16(xn @ fc1), bf16(xn @ fc2)          128 -> hidden (512), twice
//   hidden = bf16(bf16(a * bf16(sigmoid(a))) * b)     silu(a) * b
//   out    = bf16(hidden @ fc3)   (+ residual)        hidden -> 128
//
// Reference: transition_forward,
// src/foldjax/models/boltz2/models/primitives/transition.py:41-127 (the
// unchunked XLA branch :108-112); called on the pair tensor from the Pairformer
// block, src/foldjax/models/boltz2/models/pairformer.py:152-160.
//
// One tile = 128 consecutive pairs (rows of the flattened [rows][128] tensor).
// The widened form (rows x 1024) never leaves the SM: the hidden dimension is
// walked in chunks of 64, each chunk's [a | b] accumulates in TMEM, is turned
// into 64 hidden values per pair by the activation warps, goes back to shared
// memory as the A operand of the second product and is consumed there.
// The weights (384 KiB as bf16) do not fit in shared memory; they stream from
// L2 through two rings: fc1 and fc2 of a chunk (32 KiB) until its first product is through, fc3
// (16 KiB) until its second.
//
// Persistent, one CTA per SM:
//   warp 0        TMA producer of the weight chunks
//   warp 1        MMA issuer: D1[chunk] = xn . [W1c ; W2c]^T, then OUT += h . W3c^T two chunks later
//   warp 2        TMA producer of the x tiles        (warp 3 idle)
//   warps 4-7     layer norm of the x tile in place (three register-light sweeps)
//   warps 8-11    epilogue of OUT: residual fetched in whole lines before the products are waited
//                 for, sum staged in shared memory, TMA stores per warp
//   warps 12-27   activation: two groups of two warpgroups that take alternate chunks, each with a
//                 D1 and an h buffer of its own; a warpgroup turns 32 of the 64 [a | b] column pairs
//                 of every row into hidden values
// Bound: the activation (two MUFU operations per hidden unit: 1024 per pair) and
// the tensor pipe (393 kflop per pair) are within 25 % of each other; HBM moves
// 2 x 256 B per pair (x doubles as the residual when the caller adds in place). MUFU unit 68 % busy,
// tensor pipe 51 %. 1024 x 1024 pairs, hidden 512: 415 us (251 at the tensor cores' rate); 575 with
// one warpgroup for layer norm and epilogue in turn and a thread per pair's row and residual, for
// which everything else waits.
#include "host.cuh"
#include "ln.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int HC = 64;  // hidden units per chunk
constexpr int WSTAGES = 2;   // fc1 and fc2 of a chunk
constexpr int W3STAGES = 3;  // fc3 of a chunk: used two chunks after those
constexpr int XSTAGES = 2;
constexpr int TILE_BYTES = 2 * SLAB_BYTES;
constexpr int NWORK = 4;  // activation warpgroups, two per chunk parity
constexpr int THREADS = 3 * 128 + NWORK * 128;

struct Smem {
  uint8_t w12[WSTAGES][2 * SLAB_BYTES];  // fc1 and fc2 of the chunk: [128 in][64 hidden] each, MN-major
  uint8_t w3[W3STAGES][SLAB_BYTES];      // fc3 of the chunk: two boxes [64 hidden][64 out], MN-major
  uint8_t x[XSTAGES][TILE_BYTES];
  uint8_t h[2][SLAB_BYTES];              // [128 pairs][64 hidden], by chunk parity
  uint8_t out[SLAB_BYTES];               // [128 pairs][64 channels], a quarter per epilogue warp
  alignas(16) uint32_t gamma2[64], beta2[64];
  uint64_t w_full[WSTAGES], w_empty[WSTAGES], w3_full[W3STAGES], w3_empty[W3STAGES], x_full[XSTAGES], xn_full[XSTAGES], x_empty[XSTAGES];
  uint64_t d1_full[2], d1_empty[2], h_full[2], h_empty[2], out_full[2], out_empty[2];
  uint32_t tmem_base;
};
static_assert(sizeof(Smem) <= 232448, "shared memory budget");

struct Params {
  long long rows;
  uint32_t total_tiles, nchunks;  // nchunks = hidden / 64
  bool early_weights;             // the weights may be read before pdl_wait()
  const void* gamma;
  const void* beta;
  const __nv_bfloat16* residual;
  const float* row_mask;
  float eps;
  int* status;
};

// bf16(bf16(a * bf16(sigmoid(a))) * b) for two hidden units; a and b arrive as the
// fp32 accumulators and are rounded to bf16 first, like the reference's matmul output.
__device__ __forceinline__ uint32_t swiglu_bf16x2(float a0, float a1, float b0, float b1) {
  const uint32_t a = pack_bf16x2(a0, a1);
  const float2 s = sigmoid_f32x2(make_float2(bf16_lo(a), bf16_hi(a)));
  return bf16x2_mul(bf16x2_mul(a, pack_bf16x2(s.x, s.y)), pack_bf16x2(b0, b1));
}

__global__ void __launch_bounds__(THREADS, 1)
pair_transition_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w1,
                       const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_w3,
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
    tma_prefetch_desc(&tm_w1);
    tma_prefetch_desc(&tm_w2);
    tma_prefetch_desc(&tm_w3);
    for (int s = 0; s < WSTAGES; ++s) {
      mbar_init(&sm.w_full[s], 1);
      mbar_init(&sm.w_empty[s], 1);
    }
    for (int s = 0; s < W3STAGES; ++s) {
      mbar_init(&sm.w3_full[s], 1);
      mbar_init(&sm.w3_empty[s], 1);
    }
    for (int s = 0; s < XSTAGES; ++s) {
      mbar_init(&sm.x_full[s], 1);
      mbar_init(&sm.xn_full[s], 4);
      mbar_init(&sm.x_empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&sm.d1_full[a], 1);
      mbar_init(&sm.d1_empty[a], NWORK / 2 * 4);
      mbar_init(&sm.h_full[a], NWORK / 2 * 4);
      mbar_init(&sm.h_empty[a], 1);
      mbar_init(&sm.out_full[a], 1);
      mbar_init(&sm.out_empty[a], 4);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  if (!p.early_weights) pdl_wait();
  LnParam ln_param;
  if (threadIdx.x >= 128 && threadIdx.x < 256) ln_param.request(threadIdx.x < 192 ? p.gamma : p.beta, threadIdx.x & 63);
  const uint32_t nchunks = p.nchunks;
  const uint32_t n_my = (p.total_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;  // (the grid is at most total_tiles)
  const uint32_t total_n = n_my * nchunks;                                         // chunk steps of this CTA
  auto load_w12 = [&](uint32_t n, uint32_t c) {
    const uint32_t s = n % WSTAGES;
    mbar_expect_tx(&sm.w_full[s], 2 * SLAB_BYTES);
    tma_load_2d(sm.w12[s], &tm_w1, &sm.w_full[s], c * HC, 0);
    tma_load_2d(sm.w12[s] + SLAB_BYTES, &tm_w2, &sm.w_full[s], c * HC, 0);
  };
  auto load_w3 = [&](uint32_t n, uint32_t c) {
    const uint32_t s = n % W3STAGES;
    mbar_expect_tx(&sm.w3_full[s], SLAB_BYTES);
    tma_load_2d(sm.w3[s], &tm_w3, &sm.w3_full[s], 0, c * HC);
    tma_load_2d(sm.w3[s] + SLAB_BYTES / 2, &tm_w3, &sm.w3_full[s], 64, c * HC);
  };
  if (warp == 0 && lane == 0) {  // the first chunk's weights (the thread that initialised the barriers)
    load_w12(0, 0);
    load_w3(0, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sm.tmem_base;
  int status = -1;
  auto load_x = [&](uint32_t xs, uint32_t tile) {
    const int r0 = static_cast<int>(tile * 128u);
    mbar_expect_tx(&sm.x_full[xs], TILE_BYTES);
    tma_load_2d(sm.x[xs], &tm_x, &sm.x_full[xs], 0, r0);
    tma_load_2d(sm.x[xs] + SLAB_BYTES, &tm_x, &sm.x_full[xs], 64, r0);
  };
  if (p.early_weights) pdl_wait();
  if (threadIdx.x == 0) load_x(0, blockIdx.x);  // right behind the wait
  pdl_trigger();
  // TMEM: D1 (the chunk's [a | b], 128 columns) double-buffered at 0 and 128;
  // OUT (128 columns) double-buffered over tiles at 256 and 384.

  if (warp == 0) {
    if (elect_one()) {
      uint32_t c = 0;  // chunk of step n
      for (uint32_t n = 0; n < total_n; ++n) {
        if (n > 0) {
          if (!mbar_wait(&sm.w_empty[n % WSTAGES], ((n / WSTAGES) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
          load_w12(n, c);
          if (!mbar_wait(&sm.w3_empty[n % W3STAGES], ((n / W3STAGES) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
          load_w3(n, c);
        }
        if (++c == nchunks) c = 0;
      }
    }
  } else if (warp == 2) {
    if (elect_one()) {
      for (uint32_t it = 1; it < n_my; ++it) {
        const uint32_t xs = it % XSTAGES;
        if (!mbar_wait(&sm.x_empty[xs], ((it / XSTAGES) & 1) ^ 1, p.status, ST_TIMEOUT_PRODUCER)) break;
        load_x(xs, blockIdx.x + it * gridDim.x);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, 128) | UMMA_B_MN;
      uint32_t it = 0, c = 0, jt = 0, e = 0;  // tile and chunk of the first product, of the second
      // Second products follow two chunks behind, so that each activation group finds its next D1
      // ready; one behind where a tile has one chunk (two ahead would need a tile whose layer norm
      // comes after the epilogue of this one).
      const uint32_t lag = nchunks > 1 ? 2 : 1;
      for (uint32_t n = 0; n < total_n + lag; ++n) {
        if (n < total_n) {  // first product of chunk step n
          const uint32_t xs = it % XSTAGES, ws = n % WSTAGES, d = n & 1;
          if (c == 0 && !mbar_wait(&sm.xn_full[xs], (it / XSTAGES) & 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.w_full[ws], (n / WSTAGES) & 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.d1_empty[d], ((n >> 1) & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
          const uint64_t bdesc = umma_desc_mnmajor(smem_u32(sm.w12[ws]), SLAB_BYTES);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint64_t adesc = umma_desc_kmajor(smem_u32(sm.x[xs]) + (k >> 2) * SLAB_BYTES, 128);
            umma_bf16_ss(tmem_base + d * 128, umma_desc_advance(adesc, (k & 3) * 32), umma_desc_advance(bdesc, k * 2048), idesc,
                         k != 0);
          }
          umma_commit(&sm.w_empty[ws]);
          umma_commit(&sm.d1_full[d]);
          if (++c == nchunks) {
            umma_commit(&sm.x_empty[xs]);  // every first product of the tile has been issued
            c = 0;
            ++it;
          }
        }
        if (n >= lag) {  // second product of chunk step n - lag
          const uint32_t m = n - lag, ws = m % W3STAGES, hb = m & 1, tb = jt & 1;
          if (e == 0 && !mbar_wait(&sm.out_empty[tb], ((jt >> 1) & 1) ^ 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.w3_full[ws], (m / W3STAGES) & 1, p.status, ST_TIMEOUT_MMA)) break;
          if (!mbar_wait(&sm.h_full[hb], (m >> 1) & 1, p.status, ST_TIMEOUT_MMA)) break;
          tc_fence_after();
          const uint64_t adesc = umma_desc_kmajor(smem_u32(sm.h[hb]), 128);
          const uint64_t bdesc = umma_desc_mnmajor(smem_u32(sm.w3[ws]), SLAB_BYTES / 2);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ss(tmem_base + 256 + tb * 128, umma_desc_advance(adesc, k * 32), umma_desc_advance(bdesc, k * 2048),
                         idesc, (e | k) != 0);
          umma_commit(&sm.w3_empty[ws]);
          umma_commit(&sm.h_empty[hb]);
          if (++e == nchunks) {
            umma_commit(&sm.out_full[tb]);
            e = 0;
            ++jt;
          }
        }
      }
    }
  } else if (warp >= 4 && warp < 8) {
    (threadIdx.x < 192 ? sm.gamma2 : sm.beta2)[threadIdx.x & 63] = ln_param.word();
    named_barrier(1, 128);
    const int row = threadIdx.x - 128;
    for (uint32_t it = 0; it < n_my; ++it) {
      const uint32_t xs = it % XSTAGES;
      if (!mbar_wait(&sm.x_full[xs], (it / XSTAGES) & 1, p.status, ST_TIMEOUT_PROLOGUE)) break;
      ln_row_sweeps<8>(sm.x[xs], row, sm.gamma2, sm.beta2, p.eps);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.xn_full[xs]);
    }
  } else if (warp >= 8 && warp < 12) {
    const int quarter = warp & 3, row = quarter * 32 + lane;  // pair inside the tile = TMEM lane
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + 256;
    bool alive = true;
    for (uint32_t it = 0; it < n_my && alive; ++it) {
      const uint32_t tb = it & 1;
      const long long r0 = static_cast<long long>(blockIdx.x + it * gridDim.x) * 128 + quarter * 32;  // the warp's first pair
      // optional per-row mask on the update (before the residual add), rounded to the trunk dtype
      const float mkf = p.row_mask && r0 + lane < p.rows ? p.row_mask[r0 + lane] : 1.0f;
      const uint32_t mk2 = pack_bf16x2(mkf, mkf);
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {  // 64 channels at a time
        uint4 res[8];  // residual of the warp's 32 pairs, 8 lanes to a pair's 64 channels (whole lines)
        if (p.residual) {
          const long long r = r0 + (lane >> 3);
          const __nv_bfloat16* src = p.residual + r * 128 + half * 64 + (lane & 7) * 8;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            res[q] = r + 4 * q < p.rows ? *reinterpret_cast<const uint4*>(src + 512 * q) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (half == 0 && !mbar_wait(&sm.out_full[tb], (it >> 1) & 1, p.status, ST_TIMEOUT_EPILOGUE)) {
          alive = false;
          break;
        }
        if (lane == 0) tma_store_wait_read();  // the previous half has left the staging rows
        __syncwarp();
        tc_fence_after();
#pragma unroll
        for (int chunk = 0; chunk < 4; ++chunk) {
          uint32_t v[16];
          tmem_ld16(lane_addr + tb * 128 + half * 64 + chunk * 16, v);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t u[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              u[e] = pack_bf16x2(__uint_as_float(v[8 * q + 2 * e]), __uint_as_float(v[8 * q + 2 * e + 1]));
              if (p.row_mask) u[e] = bf16x2_mul(u[e], mk2);
            }
            *reinterpret_cast<uint4*>(sm.out + sw128_offset(row, chunk * 2 + q)) = make_uint4(u[0], u[1], u[2], u[3]);
          }
        }
        if (p.residual) {  // the caller's z + update, one more bf16 rounding, in the residual's arrangement
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            uint4* ptr = reinterpret_cast<uint4*>(sm.out + sw128_offset(quarter * 32 + 4 * q + (lane >> 3), lane & 7));
            uint4 u = *ptr;
            u.x = bf16x2_add(res[q].x, u.x);
            u.y = bf16x2_add(res[q].y, u.y);
            u.z = bf16x2_add(res[q].z, u.z);
            u.w = bf16x2_add(res[q].w, u.w);
            *ptr = u;
          }
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0 && r0 < p.rows) {  // rows past the end are outside the tensor and are not written
          tma_store_2d(&tm_out, sm.out + quarter * 4096, half * 64, static_cast<int>(r0));
          tma_store_commit();
        }
      }
      if (!alive) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.out_empty[tb]);
    }
    status = stores_read_and_status(lane == 0, p.status);
  } else if (warp >= 12) {
    // ---- activation: 32 columns of a and of b -> 32 hidden values, 16 at a time
    const int quarter = warp & 3, row = quarter * 32 + lane;  // pair inside the tile = TMEM lane
    const uint32_t group = (warp - 12) >> 3, half = ((warp - 12) >> 2) & 1;
    const uint32_t d1 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + group * 128 + half * 32;
    for (uint32_t n = group; n < total_n; n += 2) {
      // (a vote: each lane polls for itself, TMEM accesses take the whole warp, and all or none of it leave)
      if (!__all_sync(0xffffffffu, mbar_wait(&sm.d1_full[group], (n >> 1) & 1, p.status, ST_TIMEOUT_EPILOGUE))) break;
      tc_fence_after();
      uint32_t hv[16];
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t a[16], b[16];
        tmem_ld16(d1 + part * 16, a);
        tmem_ld16(d1 + HC + part * 16, b);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 8; ++e)
          hv[part * 8 + e] = swiglu_bf16x2(__uint_as_float(a[2 * e]), __uint_as_float(a[2 * e + 1]), __uint_as_float(b[2 * e]),
                                           __uint_as_float(b[2 * e + 1]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.d1_empty[group]);
      // this group's previous second product must have read h before it is overwritten
      if (!__all_sync(0xffffffffu, mbar_wait(&sm.h_empty[group], ((n >> 1) & 1) ^ 1, p.status, ST_TIMEOUT_EPILOGUE))) break;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(sm.h[group] + sw128_offset(row, half * 4 + q)) =
            make_uint4(hv[4 * q], hv[4 * q + 1], hv[4 * q + 2], hv[4 * q + 3]);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.h_full[group]);
    }
  }

  settle(status, p.status);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

}  // namespace
}  // namespace b200

extern "C" size_t b200tri_pair_transition_workspace_bytes(int32_t hidden) {
  if (hidden <= 0) return 0;
  return static_cast<size_t>(3) * hidden * 128 * 2 + 3 * 1024 + 1024;
}

extern "C" int b200tri_pair_transition(const b200tri_pair_transition_args* a, b200tri_stream_t stream_) {
  using namespace b200;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "pair transition: null args");
  B200_REQUIRE(a->x && a->out && a->norm_scale && a->norm_bias && a->fc1 && a->fc2 && a->fc3, B200TRI_ERR_INVALID,
               "pair transition: null pointer argument");
  B200_REQUIRE(a->rows > 0 && a->rows < (1ll << 31) - 256, B200TRI_ERR_INVALID,
               "pair transition: rows must be in [1, 2^31 - 256)");
  B200_REQUIRE(a->channels == 128, B200TRI_ERR_UNSUPPORTED, "pair transition: built for 128 channels (got %d)", a->channels);
  B200_REQUIRE(a->hidden > 0 && a->hidden % HC == 0 && a->hidden <= 4096, B200TRI_ERR_UNSUPPORTED,
               "pair transition: hidden width must be a positive multiple of 64 up to 4096 (got %d)", a->hidden);
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(a->x) | reinterpret_cast<uintptr_t>(a->out) |
                 reinterpret_cast<uintptr_t>(a->residual)) & 15) == 0,
               B200TRI_ERR_INVALID, "pair transition: x/out/residual must be 16-byte aligned");
  const size_t need = b200tri_pair_transition_workspace_bytes(a->hidden);
  B200_REQUIRE(a->workspace && a->workspace_bytes >= need, B200TRI_ERR_WORKSPACE,
               "pair transition: workspace of %zu bytes needed", need);
  int* status = device_status_word();
  B200_REQUIRE(status != nullptr, B200TRI_ERR_CUDA, "pair transition: no current CUDA device");

  // the weights are read in place; the workspace is only for one that is not 16-byte aligned
  Carver ws(a->workspace);
  const size_t w_elems = static_cast<size_t>(a->hidden) * 128;
  const void* const w_in[3] = {a->fc1, a->fc2, a->fc3};
  const void* w[3];
  for (int i = 0; i < 3; ++i) {
    const int rc = aligned_weight(w_in[i], w_elems * 2, ws.take<__nv_bfloat16>(w_elems), stream, &w[i]);
    if (rc) return rc;
  }

  CUtensorMap tm_x, tm_w1, tm_w2, tm_w3, tm_out;
  {  // the result, one box per warp: [32 pairs][64 channels]
    const uint64_t dims[2] = {128, (uint64_t)a->rows};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 32};
    int rc = make_tmap(&tm_out, a->out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    const uint64_t dims[2] = {128, (uint64_t)a->rows};
    const uint64_t str[1] = {256};
    const uint32_t box[2] = {64, 128};
    int rc = make_tmap(&tm_x, a->x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    int rc = make_weight_map(&tm_w1, w[0], 128, a->hidden, 128);
    if (rc || (rc = make_weight_map(&tm_w2, w[1], 128, a->hidden, 128))) return rc;
    if ((rc = make_weight_map(&tm_w3, w[2], a->hidden, 128, HC))) return rc;
  }
  Params p;
  p.rows = a->rows;
  p.total_tiles = static_cast<uint32_t>((a->rows + 127) / 128);
  p.early_weights = pdl_chained() && w[0] == w_in[0] && w[1] == w_in[1] && w[2] == w_in[2];
  p.nchunks = a->hidden / HC;
  p.gamma = a->norm_scale;
  p.beta = a->norm_bias;
  p.residual = static_cast<const __nv_bfloat16*>(a->residual);
  p.row_mask = a->row_mask;
  p.eps = a->eps;
  p.status = status;

  {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(pair_transition_kernel), (int)sizeof(Smem));
    if (rc) return rc;
  }
  const uint32_t sms = sm_count(), grid = p.total_tiles < sms ? p.total_tiles : sms;
  {
    TimedLaunch timed(K_PAIR_TRANSITION, stream);
    return launch(pair_transition_kernel, dim3(grid), dim3(THREADS), sizeof(Smem), stream, true, tm_x,
                  tm_w1, tm_w2, tm_w3, tm_out, p);
  }
}
