// Triangle multiplicative update, contraction stage.
//
//   t[d][i][j] = sum_{s,k} a[s][d][i][k] * b[s][d][j][k]        d = 0..127
//
// 128 independent N x N x N matrix products with both operands K-major, the
// shape tcgen05.mma consumes directly. Persistent kernel, one CTA per SM:
//   warp 0      TMA producer   (A 128x64 or 256x64 and B 256x64 or 128x64 bf16 tiles, ring of 4 or 3 stages)
//   warp 1      MMA issuer     (128x256x16 or 128x128x16 tcgen05.mma, fp32 accumulators in
//                               TMEM, two accumulators: see Cfg)
//   warps 4-11  epilogue       two warpgroups, half of the columns each: TMEM -> bf16 -> shared memory ->
//                              TMA store per warp, 32 rows x 64 columns at a time; float32 results
//                              and running sums go to global memory directly
// Tiles are walked channel by channel so the A_d/B_d panels of the channel in
// flight (2 * N*N*2 bytes) stay in L2 while all SMs work on them.
//
// Bound: large n_k, in the narrow form the operand traffic into the SM (48 KiB per k step, 768 clocks
// at 64 B/clk, against 512 of products), in the wide one an epilogue that no product overlaps (64 KiB
// for 1024 clocks of products: tensor pipe 68 % busy at n = 1024); small n_k, the epilogue.
// Algorithmic work 2*128*n_i*n_j*n_k*n_src flop. One epilogue warpgroup whose threads store 64 bytes
// of a row each (32 lines per instruction) spends 11 400 clocks on a tile of n = 200, four times its
// products and loads: 20 / 71 / 262 us at n = 203 / 500 / 1024, staged 15 / 49 / 214.
#include "host.cuh"
#include "tc.cuh"

namespace b200 {

namespace {

constexpr int BM = 128, BN_WIDE = 256, BK = 64;  // BM: rows of one accumulator
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int EPI_WARPS = 8, STAGED = 32 * 128;  // bytes a warp stages: 32 rows x 64 bf16
// H = 1: tiles of 128 rows, two accumulators in turn, so that the epilogue of one tile overlaps the
// products of the next. H = 2: tiles of 256 rows that share each k step's B, one accumulator per
// half: 64 KiB into the SM per 1024 clocks of products instead of 48 per 512, and an epilogue that
// only overlaps the loads of the next tile.
// n = 768 / 1024 / 3072: 111 / 226 / 5300 us with H = 1, 108 / 214 / 5000 with H = 2.
// BN: columns of a tile, 256, or 128 where there are no more: half the products and both epilogue warpgroups at work
// (multiplication of 77 tokens 22.9 -> 21.9 us).
template <int H, int BN>
struct Cfg {
  static constexpr int STAGE_BYTES = H * A_BYTES + BN * BK * 2, STAGES = H == 1 ? 4 : 3;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * STAGED + 1024;  // + slack for 1 KiB alignment
};
constexpr int THREADS = 128 + EPI_WARPS * 32;

struct ContractParams {
  int n_i, n_j, n_src;
  ContractTerms terms;
  int kb_per_src;  // ceil(n_k / BK)
  int tiles_m, tiles_n;
  uint32_t total_tiles;
  bool staged;  // the result leaves by TMA: it is bf16 only and a warp's 32 rows share a block
  bool out_blocked;
  bool f32_sectors;  // rows of the float32 result start on 32-byte boundaries
  const float* acc_in;
  float* out_f32;
  __nv_bfloat16* out_bf16;
  long long out_ld, out_chan_stride;
  int a_rpb, b_rpb, out_rpb;  // rows per block of the row-blocked layouts
  long long out_block_stride;
  int* status;
};

template <int H, int BN>
__global__ void __launch_bounds__(THREADS, 1)
contract_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                const __grid_constant__ CUtensorMap tm_out, const ContractParams p) {
  constexpr int STAGES = Cfg<H, BN>::STAGES, STAGE_BYTES = Cfg<H, BN>::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_base_s;

  // (through a shuffle, so that the compiler knows it to be the same in all lanes)
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_a);
    tma_prefetch_desc(&tm_b);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], EPI_WARPS / H);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_s, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  int status = -1;
  const uint32_t tmem_base = tmem_base_s;

  const int k_iters = p.n_src * p.kb_per_src;
  // (32-bit: a 64-bit division costs a role hundreds of cycles per tile)
  const uint32_t tiles_per_chan = static_cast<uint32_t>(p.tiles_m) * p.tiles_n;
  auto locate = [&](uint32_t tile, int& d, int& mi, int& nj) {
    d = tile / tiles_per_chan;
    const uint32_t rem = tile - d * tiles_per_chan;
    mi = rem / p.tiles_n;
    nj = rem - mi * p.tiles_n;
  };

  // where the producer finds a tile's operands: the first one's worked out ahead of the wait
  int src_d, a_block[H], a_row[H], b_block, b_row;
  auto origin = [&](uint32_t tile) {
    int mi, nj;
    locate(tile, src_d, mi, nj);
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const int row = (mi * H + h) * BM;
      a_block[h] = row / p.a_rpb;
      a_row[h] = row - a_block[h] * p.a_rpb;
    }
    b_block = nj * BN / p.b_rpb;
    b_row = nj * BN - b_block * p.b_rpb;
  };
  if (warp == 0) origin(blockIdx.x);
  pdl_wait();
  pdl_trigger();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool alive = true;
      for (uint32_t tile = blockIdx.x; tile < p.total_tiles && alive; tile += gridDim.x) {
        if (tile != blockIdx.x) origin(tile);
        for (int s = 0; s < p.n_src && alive; ++s) {
          for (int kb = 0; kb < p.kb_per_src; ++kb) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ST_TIMEOUT_PRODUCER)) {
              alive = false;
              break;
            }
            uint8_t* sa = smem + stage * STAGE_BYTES;
            mbar_expect_tx(&full_bar[stage], STAGE_BYTES);
            // rows are (block, row in block): a tile starts at block row0 / rpb
#pragma unroll
            for (int h = 0; h < H; ++h)
              tma_load_5d(sa + h * A_BYTES, &tm_a, &full_bar[stage], kb * BK, a_row[h], a_block[h], src_d,
                          p.terms.n ? p.terms.a[s] : s);
            tma_load_5d(sa + H * A_BYTES, &tm_b, &full_bar[stage], kb * BK, b_row, b_block, src_d,
                        p.terms.n ? p.terms.b[s] : s);
            if (++stage == STAGES) {
              stage = 0;
              phase ^= 1;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t it = 0;
      bool alive = true;
      for (uint32_t tile = blockIdx.x; tile < p.total_tiles && alive; tile += gridDim.x, ++it) {
        // (one tile's accumulator out of two in turn, or one accumulator per half)
        const uint32_t acc = it & 1, acc_phase = (H == 1 ? it >> 1 : it) & 1;
        if (!mbar_wait(&acc_empty[H == 1 ? acc : 0], acc_phase ^ 1, p.status, ST_TIMEOUT_MMA)) break;
        if (H == 2 && !mbar_wait(&acc_empty[1], acc_phase ^ 1, p.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (H == 1 ? acc * BN : 0);
        for (int ki = 0; ki < k_iters; ++ki) {
          if (!mbar_wait(&full_bar[stage], phase, p.status, ST_TIMEOUT_MMA)) {
            alive = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * STAGE_BYTES);
          const uint64_t bdesc = umma_desc_kmajor(sa + H * A_BYTES, 128);
#pragma unroll
          for (int h = 0; h < H; ++h) {
            const uint64_t adesc = umma_desc_kmajor(sa + h * A_BYTES, 128);
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_bf16_ss(d_tmem + h * BN, umma_desc_advance(adesc, k * 32), umma_desc_advance(bdesc, k * 32), idesc,
                           (ki | k) != 0);
          }
          umma_commit(&empty_bar[stage]);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (alive) umma_commit(&acc_full[H == 1 ? acc : 0]);
      }
    }
  } else if (warp >= 4) {
    const int quarter = warp & 3;  // TMEM lane quarter this warp may read
    const int group = (warp - 4) >> 2;  // which half of the tile's columns, or which of its rows
    constexpr int COLS = BN / (3 - H);   // columns of a warp
    const int first = H == 1 ? group * COLS : 0;
    uint8_t* staging = smem + STAGES * STAGE_BYTES + (warp - 4) * STAGED;
    uint32_t it = 0;
    for (uint32_t tile = blockIdx.x; tile < p.total_tiles; tile += gridDim.x, ++it) {
      int d, mi, nj;
      locate(tile, d, mi, nj);
      const uint32_t acc = H == 1 ? it & 1 : group, acc_phase = (H == 1 ? it >> 1 : it) & 1;
      if (!mbar_wait(&acc_full[H == 1 ? acc : 0], acc_phase, p.status, ST_TIMEOUT_EPILOGUE)) break;
      __syncwarp();
      tc_fence_after();
      const int row0 = (mi * H + (H == 1 ? 0 : group)) * BM + quarter * 32, row = row0 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN;
      if (p.staged) {
        const int block = row0 / p.out_rpb, in_block = row0 - block * p.out_rpb;
#pragma unroll 1
        for (int c = first; c < first + COLS; c += 64) {
          const int col0 = nj * BN + c;
          if (row0 >= p.n_i || col0 >= p.n_j) break;
          uint32_t r[2][32];
          tmem_ld32(taddr + c, r[0]);
          tmem_ld32(taddr + c + 32, r[1]);
          if (lane == 0) tma_store_wait_read();  // the staging rows are free again
          tmem_ld_wait();
          __syncwarp();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            uint32_t u[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              u[e] = pack_bf16x2(__uint_as_float(r[q >> 2][8 * (q & 3) + 2 * e]), __uint_as_float(r[q >> 2][8 * (q & 3) + 2 * e + 1]));
            *reinterpret_cast<uint4*>(staging + sw128_offset(lane, q)) = make_uint4(u[0], u[1], u[2], u[3]);
          }
          fence_proxy_async();
          __syncwarp();
          if (row0 + 32 <= p.n_i || !p.out_blocked) {
            if (lane == 0) {  // rows past n_i, and columns past n_j up to a multiple of 8, are not written
              tma_store_4d(&tm_out, staging, col0, in_block, d, block);
              tma_store_commit();
            }
          } else {  // the last block may end in rows that do not exist but lie inside the tensor
            __nv_bfloat16* dst = p.out_bf16 + static_cast<long long>(block) * p.out_block_stride +
                                 static_cast<long long>(d) * p.out_chan_stride +
                                 static_cast<long long>(in_block) * p.out_ld + col0 + (lane & 7) * 8;
            const int left = p.n_j - col0 - (lane & 7) * 8;  // columns from this lane's chunk on
            for (int rr = lane >> 3; rr < p.n_i - row0; rr += 4) {
              const uint4 u = *reinterpret_cast<const uint4*>(staging + sw128_offset(rr, lane & 7));
              if (left >= 8) {
                *reinterpret_cast<uint4*>(dst + static_cast<long long>(rr) * p.out_ld) = u;
              } else {
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int e = 0; e < 8; ++e)
                  if (e < left)
                    dst[static_cast<long long>(rr) * p.out_ld + e] =
                        __ushort_as_bfloat16(static_cast<unsigned short>((e & 1) ? (w[e >> 1] >> 16) : (w[e >> 1] & 0xffffu)));
              }
            }
            __syncwarp();
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
        continue;
      }
      const long long row_off = static_cast<long long>(row / p.out_rpb) * p.out_block_stride +
                                static_cast<long long>(d) * p.out_chan_stride +
                                static_cast<long long>(row % p.out_rpb) * p.out_ld;
#pragma unroll 1
      for (int chunk = first / 32; chunk < (first + COLS) / 32; ++chunk) {
        uint32_t r[32];
        tmem_ld32(taddr + chunk * 32, r);
        tmem_ld_wait();
        const int col0 = nj * BN + chunk * 32;
        if (row < p.n_i && col0 < p.n_j) {
          const long long off = row_off + col0;
          const bool full = (col0 + 32 <= p.n_j);
          if (p.acc_in) {
            if (full) {
              const float4* src = reinterpret_cast<const float4*>(p.acc_in + off);
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                const float4 v = src[q];
                r[4 * q + 0] = __float_as_uint(__uint_as_float(r[4 * q + 0]) + v.x);
                r[4 * q + 1] = __float_as_uint(__uint_as_float(r[4 * q + 1]) + v.y);
                r[4 * q + 2] = __float_as_uint(__uint_as_float(r[4 * q + 2]) + v.z);
                r[4 * q + 3] = __float_as_uint(__uint_as_float(r[4 * q + 3]) + v.w);
              }
            } else {
#pragma unroll
              for (int q = 0; q < 32; ++q)
                if (col0 + q < p.n_j) r[q] = __float_as_uint(__uint_as_float(r[q]) + p.acc_in[off + q]);
            }
          }
          if (p.out_f32) {
            if (full) {
              float4* dst = reinterpret_cast<float4*>(p.out_f32 + off);
              if (p.f32_sectors) {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                  store_sector(dst + 2 * q, make_uint4(r[8 * q], r[8 * q + 1], r[8 * q + 2], r[8 * q + 3]),
                               make_uint4(r[8 * q + 4], r[8 * q + 5], r[8 * q + 6], r[8 * q + 7]));
              } else {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                  dst[q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]),
                                       __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
              }
            } else {
#pragma unroll
              for (int q = 0; q < 32; ++q)
                if (col0 + q < p.n_j) p.out_f32[off + q] = __uint_as_float(r[q]);
            }
          }
          if (p.out_bf16) {
            if (full) {
              uint4* dst = reinterpret_cast<uint4*>(p.out_bf16 + off);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                uint4 v;
                v.x = pack_bf16x2(__uint_as_float(r[8 * q + 0]), __uint_as_float(r[8 * q + 1]));
                v.y = pack_bf16x2(__uint_as_float(r[8 * q + 2]), __uint_as_float(r[8 * q + 3]));
                v.z = pack_bf16x2(__uint_as_float(r[8 * q + 4]), __uint_as_float(r[8 * q + 5]));
                v.w = pack_bf16x2(__uint_as_float(r[8 * q + 6]), __uint_as_float(r[8 * q + 7]));
                dst[q] = v;
              }
            } else {
#pragma unroll
              for (int q = 0; q < 32; ++q)
                if (col0 + q < p.n_j) p.out_bf16[off + q] = __float2bfloat16_rn(__uint_as_float(r[q]));
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
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

extern "C" int b200tri_trimul_contract(const b200tri_trimul_contract_args* a, b200tri_stream_t stream) {
  return b200::contract_launch(a, 128, b200::ContractTerms{}, false, reinterpret_cast<cudaStream_t>(stream));
}

int b200::contract_launch(const b200tri_trimul_contract_args* a, int channels, const ContractTerms& terms, bool pad_is_scratch,
                          cudaStream_t stream) {
  B200_REQUIRE(a != nullptr, B200TRI_ERR_INVALID, "contract: null args");
  B200_REQUIRE(a->a && a->b, B200TRI_ERR_INVALID, "contract: null operand");
  B200_REQUIRE(a->out_f32 || a->out_bf16, B200TRI_ERR_INVALID, "contract: no output buffer");
  B200_REQUIRE(a->n_i > 0 && a->n_j > 0 && a->n_k > 0 && a->n_src > 0, B200TRI_ERR_INVALID,
               "contract: sizes must be positive (n_i=%d n_j=%d n_k=%d n_src=%d)", a->n_i, a->n_j, a->n_k, a->n_src);
  B200_REQUIRE(a->a_ld % 8 == 0 && a->b_ld % 8 == 0 && a->out_ld % 8 == 0 && a->a_chan_stride % 8 == 0 &&
                   a->b_chan_stride % 8 == 0 && a->a_src_stride % 8 == 0 && a->b_src_stride % 8 == 0 &&
                   a->out_chan_stride % 8 == 0,
               B200TRI_ERR_INVALID, "contract: pitches and strides must be multiples of 8 elements");
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a->out_bf16) & 15) == 0 && (reinterpret_cast<uintptr_t>(a->out_f32) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(a->acc_in) & 15) == 0,
               B200TRI_ERR_INVALID, "contract: output pointers must be 16-byte aligned");
  int* status = device_status_word();
  B200_REQUIRE(status != nullptr, B200TRI_ERR_CUDA, "contract: no current CUDA device");

  // Row-blocked operands: rows_per_block 0 (or >= the row count) means one block.
  // A blocked operand needs blocks that tile the kernel's 128- / 256-row tiles.
  auto blocking = [](int32_t rpb, int32_t n, int tile, int* rows, uint32_t* box_r, uint32_t* box_b, uint64_t* blocks) {
    if (rpb <= 0 || rpb >= n) {
      *rows = n;
      *box_r = static_cast<uint32_t>(tile);
      *box_b = 1;
      *blocks = 1;
      return true;
    }
    if (rpb % tile != 0 && tile % rpb != 0) return false;
    *rows = rpb;
    *box_r = static_cast<uint32_t>(rpb < tile ? rpb : tile);
    *box_b = static_cast<uint32_t>(tile / static_cast<int>(*box_r));
    *blocks = static_cast<uint64_t>((n + rpb - 1) / rpb);
    return true;
  };
  int a_rows, b_rows;
  uint32_t a_box_r, a_box_b, b_box_r, b_box_b;
  uint64_t a_blocks, b_blocks;
  B200_REQUIRE(blocking(a->a_rows_per_block, a->n_i, BM, &a_rows, &a_box_r, &a_box_b, &a_blocks) &&
                   blocking(a->b_rows_per_block, a->n_j, BN_WIDE, &b_rows, &b_box_r, &b_box_b, &b_blocks),
               B200TRI_ERR_INVALID, "contract: rows_per_block must divide or be a multiple of the tile rows (128 for a, 256 for b)");
  const int bn = a->n_j <= BN_WIDE / 2 ? BN_WIDE / 2 : BN_WIDE;
  blocking(a->b_rows_per_block, a->n_j, bn, &b_rows, &b_box_r, &b_box_b, &b_blocks);  // (what tiles 256 rows tiles 128)
  B200_REQUIRE(a->a_block_stride % 8 == 0 && a->b_block_stride % 8 == 0 && a->out_block_stride % 8 == 0,
               B200TRI_ERR_INVALID, "contract: block strides must be multiples of 8 elements");
  int planes = a->n_src;  // planes of an operand: one per source, or one per piece
  if (terms.n) {
    planes = 1;
    for (int t = 0; t < terms.n; ++t) {
      planes = terms.a[t] >= planes ? terms.a[t] + 1 : planes;
      planes = terms.b[t] >= planes ? terms.b[t] + 1 : planes;
    }
  }
  CUtensorMap tm_a, tm_b;
  {
    const uint64_t dims[5] = {(uint64_t)a->n_k, (uint64_t)a_rows, a_blocks, (uint64_t)channels, (uint64_t)planes};
    const uint64_t str[4] = {(uint64_t)a->a_ld * 2, (uint64_t)(a_blocks > 1 ? a->a_block_stride : a->a_chan_stride * channels) * 2,
                             (uint64_t)a->a_chan_stride * 2,
                             (uint64_t)(planes > 1 ? a->a_src_stride : a->a_chan_stride * channels) * 2};
    const uint32_t box[5] = {BK, a_box_r, a_box_b, 1, 1};
    int rc = make_tmap(&tm_a, a->a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  {
    const uint64_t dims[5] = {(uint64_t)a->n_k, (uint64_t)b_rows, b_blocks, (uint64_t)channels, (uint64_t)planes};
    const uint64_t str[4] = {(uint64_t)a->b_ld * 2, (uint64_t)(b_blocks > 1 ? a->b_block_stride : a->b_chan_stride * channels) * 2,
                             (uint64_t)a->b_chan_stride * 2,
                             (uint64_t)(planes > 1 ? a->b_src_stride : a->b_chan_stride * channels) * 2};
    const uint32_t box[5] = {BK, b_box_r, b_box_b, 1, 1};
    int rc = make_tmap(&tm_b, a->b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  const int out_rows = a->out_rows_per_block > 0 && a->out_rows_per_block < a->n_i ? a->out_rows_per_block : a->n_i;
  const int out_blocks = (a->n_i + out_rows - 1) / out_rows;
  const bool staged = a->out_bf16 && !a->out_f32 && !a->acc_in && (out_blocks == 1 || out_rows % 32 == 0) &&
                      (pad_is_scratch || a->n_j % 8 == 0);
  CUtensorMap tm_out = tm_a;  // (unused without staging)
  if (staged) {
    const uint64_t dims[4] = {(uint64_t)a->n_j, (uint64_t)out_rows, (uint64_t)channels, (uint64_t)out_blocks};
    const uint64_t str[3] = {(uint64_t)a->out_ld * 2, (uint64_t)a->out_chan_stride * 2,
                             (uint64_t)(out_blocks > 1 ? a->out_block_stride : a->out_chan_stride * channels) * 2};
    const uint32_t box[4] = {64, 32, 1, 1};
    int rc = make_tmap(&tm_out, a->out_bf16, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, dims, str, box, Swz::B128);
    if (rc) return rc;
  }
  ContractParams p;
  p.staged = staged;
  p.out_blocked = out_blocks > 1;
  p.n_i = a->n_i;
  p.n_j = a->n_j;
  p.n_src = terms.n ? terms.n : a->n_src;
  p.terms = terms;
  p.kb_per_src = (a->n_k + BK - 1) / BK;
  p.tiles_n = (a->n_j + bn - 1) / bn;
  // Tiles of 128 or 256 rows, whichever is through first: rounds over the SMs times the clocks of a
  // tile (loads, with the epilogue behind them where it is longer; products and epilogue).
  const long long sms = sm_count(), kb = static_cast<long long>(p.n_src) * p.kb_per_src;
  auto tiles_of = [&](int rows) { return static_cast<long long>(channels) * ((a->n_i + rows - 1) / rows) * p.tiles_n; };
  const long long narrow = (tiles_of(BM) + sms - 1) / sms * (kb * 768 > 3000 ? kb * 768 : 3000);
  const long long wide = (tiles_of(2 * BM) + sms - 1) / sms * (kb * 1024 + 3500);
  const int halves = bn == BN_WIDE && wide < narrow ? 2 : 1;
  p.tiles_m = (a->n_i + halves * BM - 1) / (halves * BM);
  const long long tiles = tiles_of(halves * BM);
  B200_REQUIRE(tiles < (1ll << 31), B200TRI_ERR_UNSUPPORTED, "contract: too many tiles (%lld)", tiles);
  p.total_tiles = static_cast<uint32_t>(tiles);
  p.acc_in = a->acc_in;
  p.out_f32 = a->out_f32;
  p.f32_sectors = (reinterpret_cast<uintptr_t>(a->out_f32) & 31) == 0 &&
                  (a->out_ld | a->out_chan_stride | a->out_block_stride) % 8 == 0;
  p.out_bf16 = static_cast<__nv_bfloat16*>(a->out_bf16);
  p.out_ld = a->out_ld;
  p.out_chan_stride = a->out_chan_stride;
  p.a_rpb = a_rows;
  p.b_rpb = b_rows;
  p.out_rpb = out_rows;
  p.out_block_stride = a->out_block_stride;
  p.status = status;

  const long long grid = tiles < sms ? tiles : sms;
  auto go = [&](auto kernel, int smem) {
    const int rc = ensure_smem_limit(reinterpret_cast<const void*>(kernel), smem);
    if (rc) return rc;
    TimedLaunch timed(K_TRIMUL_CONTRACT, stream);
    return launch(kernel, dim3(static_cast<unsigned>(grid)), dim3(THREADS), smem, stream, true, tm_a, tm_b, tm_out, p);
  };
  if (bn < BN_WIDE) return go(contract_kernel<1, BN_WIDE / 2>, Cfg<1, BN_WIDE / 2>::SMEM_BYTES);
  return halves == 2 ? go(contract_kernel<2, BN_WIDE>, Cfg<2, BN_WIDE>::SMEM_BYTES)
                     : go(contract_kernel<1, BN_WIDE>, Cfg<1, BN_WIDE>::SMEM_BYTES);
}
