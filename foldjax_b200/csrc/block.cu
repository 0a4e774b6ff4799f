// One Pairformer block - or a whole stack of them - as a single call.
//
// Reference: pairformer_layer_forward, src/foldjax/models/boltz2/models/trunk_blocks/
// pairformer.py:100-206, and the lax.scan over stacked layer parameters that drives it
// (pairformer.py:30-100, src/foldjax/models/_stacking.py). Op order and residuals:
//
//   z += tri_mul_out(z);  z += tri_mul_in(z);  z += tri_att_start(z);  z += tri_att_end(z)
//   z += transition_z(z)
//   s += attention_pair_bias(LN(s), z, mask, k_in = LN(s));  s += transition_s(s)
//
// The pair track is bf16 on the tensor cores (the entry points of this library, residual adds
// fused into their output stages); the single track is float32, as the reference promotes it
// (pairformer.py:182-206), with bf16 parameters. One call per block removes the per-op host
// round trips; one call per trunk replaces the scan.
#include <cuda_bf16.h>

#include <optional>

#include "host.cuh"
#include "single.cuh"

namespace b200 {
namespace {

// dst[pair][:] = mask[pair] != 0 ? src[pair][:] : 0 for 128-channel bf16 pairs, one thread per
// 16-byte chunk. With src == dst only the dropped pairs are written. The pair gate of
// Protenix's block: z * pair_valid (protenix/models/trunk_blocks/pairformer.py:71-100).
__global__ void gate_pairs_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, const float* __restrict__ mask,
                                  long long pairs) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= pairs * 16) return;
  const bool keep = mask[idx >> 4] != 0.f;
  if (!keep)
    dst[idx] = make_uint4(0u, 0u, 0u, 0u);
  else if (src != dst)
    dst[idx] = src[idx];
}

__global__ void fill_kernel(float* __restrict__ p, long long total, float v) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < total) p[i] = v;
}

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

struct Plan {
  size_t w, sub, sub_bytes, sn, partial, h, att, fc[3], ones, total;
};

// Up to this many tokens the pair track's stage kernels have one tile per SM (as many as tokens, a
// contraction 128) and leave SMs over for what runs on the side stream. The attention core does not:
// 4 * ceil(n / 3) items are more than the SMs from n = 109 on, and what meets it there delays it (17
// instead of 12 us at n = 128). All in all the pair bias aside gains at every such size, 24 blocks,
// us, n = 48 / 97 / 112 / 128: 2850 / 3195 / 3439 / 3669 without, 2730 / 3063 / 3287 / 3337 with, attention
// first 2884 / 3213 / 3418 / 3471 and 2754 / 3066 / 3264 / 3395. With more tokens a row of pairs takes two
// tiles, and the stage kernels fill every SM.
constexpr int LEFT_OVER_UP_TO = 128;
bool leaves_sms(int n) { return n <= LEFT_OVER_UP_TO; }
// The second buffer that blocks of a stack end in where the workspace has room for it, behind the plan's total.
size_t second_end_bytes(int n) { return (static_cast<size_t>(n) * n * 128 * 2 + 1023) / 1024 * 1024; }

Plan plan(int n, int c_s, int heads_s, int hidden_z, int hidden_s, bool single) {
  Plan p = {};
  Offsets o;
  p.w = o.take(static_cast<size_t>(n) * n * 128 * 2);
  size_t sub = b200tri_trimul_workspace_bytes(n);
  const size_t cand[2] = {b200tri_triatt_workspace_bytes(n), b200tri_pair_transition_workspace_bytes(hidden_z)};
  for (size_t c : cand) sub = c > sub ? c : sub;
  p.sub_bytes = sub;
  p.sub = o.take(sub);
  if (single) {
    const size_t act = static_cast<size_t>(n) * c_s;
    p.sn = o.take(act * 2 * 3);
    p.partial = o.take(act * 4 * SINGLE_MAX_SPLITS);
    p.h = o.take(static_cast<size_t>(n) * round_up(hidden_s, 8) * 2 * 3);
    p.att = o.take(single_attention_work(n, c_s, heads_s).total);
    p.fc[0] = o.take(tma_weight_bytes(c_s, hidden_s));
    p.fc[1] = o.take(tma_weight_bytes(c_s, hidden_s));
    p.fc[2] = o.take(tma_weight_bytes(hidden_s, c_s));
    p.ones = o.take(static_cast<size_t>(n) * 4);
  }
  p.total = o.total();
  return p;
}

const void* leaf(const void* base, int layer, size_t elems) {
  return base ? static_cast<const uint8_t*>(base) + static_cast<size_t>(layer) * elems * 2 : nullptr;
}

// Block `layer` of parameters stacked leaf by leaf with a leading layer axis ([L, ...] bf16).
b200tri_pairformer_block_params unstack(const b200tri_pairformer_block_params& s, int layer, int c_s, int heads_s) {
  b200tri_pairformer_block_params p = s;
  auto mul = [&](b200tri_trimul_params& d, const b200tri_trimul_params& b) {
    d.norm_in_scale = leaf(b.norm_in_scale, layer, 128);
    d.norm_in_bias = leaf(b.norm_in_bias, layer, 128);
    d.p_in = leaf(b.p_in, layer, 128 * 256);
    d.g_in = leaf(b.g_in, layer, 128 * 256);
    d.norm_out_scale = leaf(b.norm_out_scale, layer, 128);
    d.norm_out_bias = leaf(b.norm_out_bias, layer, 128);
    d.p_out = leaf(b.p_out, layer, 128 * 128);
    d.g_out = leaf(b.g_out, layer, 128 * 128);
  };
  auto att = [&](b200tri_triatt_params& d, const b200tri_triatt_params& b) {
    d.norm_scale = leaf(b.norm_scale, layer, 128);
    d.norm_bias = leaf(b.norm_bias, layer, 128);
    d.w_bias = leaf(b.w_bias, layer, 128 * 4);
    d.w_q = leaf(b.w_q, layer, 128 * 128);
    d.w_k = leaf(b.w_k, layer, 128 * 128);
    d.w_v = leaf(b.w_v, layer, 128 * 128);
    d.w_g = leaf(b.w_g, layer, 128 * 128);
    d.w_o = leaf(b.w_o, layer, 128 * 128);
  };
  auto trn = [&](b200tri_transition_params& d, const b200tri_transition_params& b, size_t c) {
    d.norm_scale = leaf(b.norm_scale, layer, c);
    d.norm_bias = leaf(b.norm_bias, layer, c);
    d.fc1 = leaf(b.fc1, layer, c * b.hidden);
    d.fc2 = leaf(b.fc2, layer, c * b.hidden);
    d.fc3 = leaf(b.fc3, layer, c * b.hidden);
  };
  mul(p.tri_mul_out, s.tri_mul_out);
  mul(p.tri_mul_in, s.tri_mul_in);
  att(p.tri_att_start, s.tri_att_start);
  att(p.tri_att_end, s.tri_att_end);
  trn(p.transition_z, s.transition_z, 128);
  p.pre_norm_s_scale = leaf(s.pre_norm_s_scale, layer, c_s);
  p.pre_norm_s_bias = leaf(s.pre_norm_s_bias, layer, c_s);
  const size_t cc = static_cast<size_t>(c_s) * c_s;
  p.attention.proj_q = leaf(s.attention.proj_q, layer, cc);
  p.attention.proj_q_bias = leaf(s.attention.proj_q_bias, layer, c_s);
  p.attention.proj_k = leaf(s.attention.proj_k, layer, cc);
  p.attention.proj_v = leaf(s.attention.proj_v, layer, cc);
  p.attention.proj_g = leaf(s.attention.proj_g, layer, cc);
  p.attention.proj_z_norm_scale = leaf(s.attention.proj_z_norm_scale, layer, 128);
  p.attention.proj_z_norm_bias = leaf(s.attention.proj_z_norm_bias, layer, 128);
  p.attention.proj_z = leaf(s.attention.proj_z, layer, 128 * static_cast<size_t>(heads_s));
  p.attention.proj_o = leaf(s.attention.proj_o, layer, cc);
  trn(p.transition_s, s.transition_s, c_s);
  return p;
}

}  // namespace
}  // namespace b200

using namespace b200;

extern "C" size_t b200tri_pairformer_workspace_bytes(int32_t n, int32_t c_s, int32_t heads_s, int32_t hidden_z,
                                                     int32_t hidden_s) {
  if (n <= 0 || hidden_z <= 0) return 0;
  return plan(n, c_s, heads_s, hidden_z, hidden_s, c_s > 0).total + 1024;
}

extern "C" size_t b200tri_pairformer_stack_workspace_bytes(int32_t n, int32_t c_s, int32_t heads_s, int32_t hidden_z,
                                                           int32_t hidden_s, int32_t n_blocks) {
  const size_t least = b200tri_pairformer_workspace_bytes(n, c_s, heads_s, hidden_z, hidden_s);
  return least && n_blocks > 1 && c_s > 0 && leaves_sms(n) ? least + second_end_bytes(n) : least;
}

extern "C" int b200tri_pairformer_forward(const b200tri_pairformer_args* a, b200tri_stream_t stream_) {
  B200_REQUIRE(a != nullptr && a->params != nullptr, B200TRI_ERR_INVALID, "pairformer: null args or params");
  B200_REQUIRE(a->n > 0 && a->n_blocks >= 1, B200TRI_ERR_INVALID, "pairformer: n and n_blocks must be positive");
  B200_REQUIRE(a->z_in && a->z_out, B200TRI_ERR_INVALID, "pairformer: z_in/z_out must not be null");
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(a->z_in) | reinterpret_cast<uintptr_t>(a->z_out)) & 15) == 0, B200TRI_ERR_INVALID,
               "pairformer: z_in/z_out must be 16-byte aligned");
  const bool single = a->s_in != nullptr;
  B200_REQUIRE(!single || (a->s_out && a->c_s > 0 && a->heads_s > 0), B200TRI_ERR_INVALID,
               "pairformer: the single track needs s_out, c_s and heads_s");
  const b200tri_pairformer_block_params& first = a->params[0];
  int hidden_z = 0, hidden_s = 0;  // of the widest block: the scratch is shared by all of them
  for (int layer = 0; layer < (a->stacked ? 1 : a->n_blocks); ++layer) {
    const int hz = a->params[layer].transition_z.hidden, hs = a->params[layer].transition_s.hidden;
    B200_REQUIRE(hz > 0 && (!single || hs > 0), B200TRI_ERR_INVALID, "pairformer: transition widths missing");
    hidden_z = hz > hidden_z ? hz : hidden_z;
    hidden_s = single && hs > hidden_s ? hs : hidden_s;
  }
  B200_REQUIRE(!single || (a->heads_s <= 16 && a->c_s == a->heads_s * 24), B200TRI_ERR_UNSUPPORTED,
               "pairformer: the single track is built for up to 16 heads of width 24 (got c_s %d, %d heads)", a->c_s,
               a->heads_s);
  const Plan pl = plan(a->n, a->c_s, a->heads_s, hidden_z, hidden_s, single);
  B200_REQUIRE(a->workspace && a->workspace_bytes >= pl.total, B200TRI_ERR_WORKSPACE,
               "pairformer: workspace of %zu bytes needed, got %zu", pl.total, a->workspace_bytes);
  B200_REQUIRE((reinterpret_cast<uintptr_t>(a->workspace) & 1023) == 0, B200TRI_ERR_INVALID,
               "pairformer: workspace must be 1024-byte aligned");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  uint8_t* ws = static_cast<uint8_t*>(a->workspace);
  void* w = ws + pl.w;
  const int n = a->n, c_s = a->c_s;
  const float* token_mask = a->mask;
  if (single && !token_mask) {
    float* ones = reinterpret_cast<float*>(ws + pl.ones);
    count_launch();
    fill_kernel<<<(n + 255) / 256, 256, 0, stream>>>(ones, n, 1.0f);
    B200_CUDA_OK(cudaGetLastError());
    token_mask = ones;
  }

  const void* z_cur = a->z_in;
  const long long pairs = static_cast<long long>(n) * n;
  const bool gate = a->pair_gate != 0 && a->pair_mask != nullptr;
  auto gate_pairs = [&](const void* src, void* dst) -> int {
    count_launch();
    gate_pairs_kernel<<<static_cast<unsigned>((pairs * 16 + 255) / 256), 256, 0, stream>>>(
        static_cast<const uint4*>(src), static_cast<uint4*>(dst), a->pair_mask, pairs);
    B200_CUDA_OK(cudaGetLastError());
    return B200TRI_OK;
  };
  auto params_of = [&](int layer) { return a->stacked ? unstack(first, layer, c_s, a->heads_s) : a->params[layer]; };
  int rc;

  // The single track is float32: s += attention(LN(s), z), s += transition(s), each sum taken by
  // the row kernel that also normalises the rows for the product behind it. The pair bias is its
  // only step that reads z, so in a stack everything else of a block's single track - six
  // launches that fill a few SMs each - runs on a side stream beside the next block's pair track,
  // and the first block's q, k, v and gate beside its own. 48 blocks at n = 128: 9.3 -> 8.2 ms, and
  // with the pair bias aside too (below) 7.3 -> 6.6.
  auto attention_args = [&](const b200tri_pairformer_block_params& P) {
    b200tri_attention_pair_bias_args t = {};
    t.n = n;
    t.c_s = c_s;
    t.c_z = 128;
    t.heads = a->heads_s;
    t.eps = a->eps;
    t.inf = a->att_inf;
    t.z = a->z_out;
    t.mask = token_mask;
    t.proj_q = P.attention.proj_q;
    t.proj_q_bias = P.attention.proj_q_bias;
    t.proj_k = P.attention.proj_k;
    t.proj_v = P.attention.proj_v;
    t.proj_g = P.attention.proj_g;
    t.proj_z_norm_scale = P.attention.proj_z_norm_scale;
    t.proj_z_norm_bias = P.attention.proj_z_norm_bias;
    t.proj_z = P.attention.proj_z;
    t.proj_o = P.attention.proj_o;
    return t;
  };
  __nv_bfloat16* sn = reinterpret_cast<__nv_bfloat16*>(ws + pl.sn);
  float* partial = reinterpret_cast<float*>(ws + pl.partial);
  __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(ws + pl.h);
  uint8_t* att = ws + pl.att;
  RowArgs row = {};
  row.rows = n;
  row.c = c_s;
  row.eps = a->eps;
  std::optional<SideStream> lease;
  if (single) {
    // (One block alone has its projection to overlap, us a call, calls in a row, without and with: 96 tokens 155.5 / 151, 128
    // 169.1 / 163.1, 203 272.1 / 267.6, 300 487.2 / 482.6, 512 level.)
    lease.emplace(stream);
    const b200tri_pairformer_block_params P = params_of(0);
    row.base = a->s_in;
    row.scale = P.pre_norm_s_scale;
    row.bias = P.pre_norm_s_bias;
    row.pieces = sn;
    cudaStream_t st = lease->stream ? lease->stream : stream;
    const b200tri_attention_pair_bias_args t = attention_args(P);
    if ((rc = lease->fork()) || (rc = launch_row_norm(row, st, false)) || (rc = single_project(&t, sn, sn, att, st)) ||
        (rc = lease->mark()))
      return rc;
  }

  // Where the pair track leaves SMs over, the pair bias is on the side stream as well, on those SMs,
  // while the next block's pair track runs on z in a buffer of its own: blocks end in z_out and w2 in
  // turn, the last one in z_out. (In one buffer, with the wait for the pair bias ahead of the next
  // block's second update, 24 blocks took 3430 instead of 3340 us at n = 128 and 3040 instead of 3075 at 100.)
  const bool bias_aside = single && lease->stream && leaves_sms(n) && sm_count() >= LEFT_OVER_UP_TO + 16 &&
                          a->workspace_bytes >= pl.total + second_end_bytes(n);
  void* w2 = bias_aside ? ws + pl.total : nullptr;
  const int over = bias_aside ? sm_count() - LEFT_OVER_UP_TO : 0;

  PdlChain chain(false);
  for (int layer = 0; layer < a->n_blocks; ++layer) {
    const b200tri_pairformer_block_params P = params_of(layer);
    void* z_end = bias_aside && (a->n_blocks - 1 - layer) % 2 ? w2 : a->z_out;
    // ---- pair track: the four triangle updates ping-pong between z_out and w (the first one
    // reads the caller's z_in), residual adds fused; with the pair gate, dropped pairs are
    // zeroed before the first update and after every update
    if (gate && layer == 0) {
      if ((rc = gate_pairs(z_cur, a->z_out))) return rc;  // a gated copy, or in place when they alias
      z_cur = a->z_out;
    }
    for (int k = 0; k < 4; ++k) {
      // Boltz-2 / Protenix / OpenFold3 default: multiplications first; attention_first swaps the halves
      const int op = a->attention_first ? (k + 2) % 4 : k;  // 0 out, 1 in, 2 start, 3 end
      void* dst = z_cur == w ? z_end : w;
      if (op < 2) {
        const b200tri_trimul_params& m = op == 0 ? P.tri_mul_out : P.tri_mul_in;
        b200tri_trimul_args t = {};
        t.n = n;
        t.incoming = op;
        t.eps = a->eps;
        t.x = z_cur;
        t.mask = a->pair_mask;
        t.norm_in_scale = m.norm_in_scale;
        t.norm_in_bias = m.norm_in_bias;
        t.p_in = m.p_in;
        t.g_in = m.g_in;
        t.norm_out_scale = m.norm_out_scale;
        t.norm_out_bias = m.norm_out_bias;
        t.p_out = m.p_out;
        t.g_out = m.g_out;
        t.residual = t.x;
        t.out = dst;
        t.workspace = ws + pl.sub;
        t.workspace_bytes = pl.sub_bytes;
        if ((rc = b200tri_trimul_forward(&t, stream_))) return rc;
      } else {
        const b200tri_triatt_params& m = op == 2 ? P.tri_att_start : P.tri_att_end;
        b200tri_triatt_args t = {};
        t.n = n;
        t.starting = op == 2;
        t.heads = 4;
        t.head_dim = 32;
        t.inf = a->tri_inf;
        t.eps = a->eps;
        t.x = z_cur;
        t.mask = a->pair_mask;
        t.norm_scale = m.norm_scale;
        t.norm_bias = m.norm_bias;
        t.w_bias = m.w_bias;
        t.w_q = m.w_q;
        t.w_k = m.w_k;
        t.w_v = m.w_v;
        t.w_g = m.w_g;
        t.w_o = m.w_o;
        t.residual = t.x;
        t.out = dst;
        t.workspace = ws + pl.sub;
        t.workspace_bytes = pl.sub_bytes;
        if ((rc = b200tri_triatt_forward(&t, stream_))) return rc;
      }
      chain.set();
      if (gate && (rc = gate_pairs(dst, dst))) return rc;
      z_cur = dst;
    }
    // four updates from wherever the block before ended end in z_end
    {
      b200tri_pair_transition_args t = {};
      t.rows = static_cast<int64_t>(n) * n;
      t.channels = 128;
      t.hidden = P.transition_z.hidden;
      t.eps = a->eps;
      t.x = z_end;
      t.norm_scale = P.transition_z.norm_scale;
      t.norm_bias = P.transition_z.norm_bias;
      t.fc1 = P.transition_z.fc1;
      t.fc2 = P.transition_z.fc2;
      t.fc3 = P.transition_z.fc3;
      t.residual = z_end;
      t.out = z_end;  // row-local: in place
      t.workspace = ws + pl.sub;
      t.workspace_bytes = pl.sub_bytes;
      t.row_mask = a->mask_transition ? a->pair_mask : nullptr;
      if ((rc = b200tri_pair_transition(&t, stream_))) return rc;
      if (gate && (rc = gate_pairs(z_end, z_end))) return rc;
    }
    z_cur = z_end;
    if (!single) continue;
    SideStream& side = *lease;

    // ---- single track; the last block's is on the caller's stream
    const bool last = layer + 1 == a->n_blocks, forked = side.stream != nullptr;
    b200tri_attention_pair_bias_args t = attention_args(P);
    t.z = z_end;
    cudaStream_t st = last || !forked ? stream : side.stream;
    if (bias_aside && !last) {
      // (z of the block before, which the next block overwrites, has been read)
      if (layer > 0 && (rc = side.join_early())) return rc;
      if ((rc = side.fork())) return rc;
      SmReserve others(sm_count() - over);
      if ((rc = single_pair_bias(&t, att, st, false)) || (rc = side.mark_early())) return rc;
    } else {
      if ((rc = side.join()) || (rc = single_pair_bias(&t, att, stream, !forked))) return rc;
      if (!last && (rc = side.fork())) return rc;
    }
    int splits = 1;
    if ((rc = single_attend(&t, att, partial, &splits, st, last || !forked))) return rc;
    row.base = layer == 0 ? a->s_in : a->s_out;
    row.partial = partial;
    row.splits = splits;
    row.row_mask = gate ? token_mask : nullptr;
    row.scale = P.transition_s.norm_scale;
    row.bias = P.transition_s.norm_bias;
    row.sum_out = a->s_out;
    row.pieces = sn;
    if ((rc = launch_row_norm(row, st, true))) return rc;
    // transition_s: LN -> fc1 | fc2 -> silu(fc1) * fc2 -> fc3, added to s (transition.py:99-112)
    const int hid = P.transition_s.hidden;
    const long long hp = round_up(hid, 8);
    if ((rc = launch_swiglu(sn, n, c_s, P.transition_s.fc1, P.transition_s.fc2, hid, ws + pl.fc[0], ws + pl.fc[1], h, hp, st,
                            true)))
      return rc;
    if ((rc = launch_linear_partial(h, hp, n, hid, P.transition_s.fc3, c_s, ws + pl.fc[2], partial, &splits, st, true)))
      return rc;
    row.base = a->s_out;
    row.splits = splits;
    if (last) {
      row.pieces = nullptr;
      if ((rc = launch_row_norm(row, st, true))) return rc;
      break;
    }
    const b200tri_pairformer_block_params next = params_of(layer + 1);
    row.scale = next.pre_norm_s_scale;
    row.bias = next.pre_norm_s_bias;
    if ((rc = launch_row_norm(row, st, true))) return rc;
    const b200tri_attention_pair_bias_args t_next = attention_args(next);
    if ((rc = single_project(&t_next, sn, sn, att, st)) || (rc = side.mark())) return rc;
  }
  return B200TRI_OK;
}
