// The host side of a step in native code: which kernel takes which product, the gated feed-forward,
// one layer's attention, and the whole stack of layers of a step (see oi_api.h).
//
// The reference's step is native host code that launches one kernel after the other
// (pegainfer-qwen3/src/executor.rs:365-620, unified_forward.rs:383-611); so is this. Everything here only
// chooses and launches: the kernels are the ones in the other files of this folder, called through
// their checked entry points.
#include "oi_api.h"

namespace {

int g_opt[OI_OPT_COUNT] = {0, 0, 0, 0, 129, 0};
constexpr int kDecodeMaxRows = 32;    // rows up to which the streaming product takes a product
constexpr int kSkinnyMaxRows = 16;
constexpr int kFusedMinRows = 128;    // rows from which gate/up forms the activation in the tcgen05 product's epilogue
constexpr int kPair = 0;              // tile_n value that stands for 256 x 256 tiles of a pair of CTAs

// operands that TMA can fetch: rows contiguous in k, 16-byte aligned bases and row strides
bool tma_ok(const void* x, long long ldx, const void* w, long long ldw, int K) {
  return K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0;
}

// This host thread launches a step whose experts are chosen by scores (oi_streamed_products).
thread_local int t_streamed = 0;

// How many K slices (CTAs per cluster) the streaming kernel uses: one when the tiles of 128 weight rows alone
// fill the GPU, else the fewest slices that give every SM a CTA, each slice at least two k blocks long, while all CTAs run at
// once: two fit on an SM, but clusters of 8 only 33 at a time (264 CTAs), of 4 some 70 (280; with 284 it depends on the kernel
// before), and what is left over runs alone.
// Measured on B200 at M = 8 (us, inside a CUDA graph): N 6144 K 4096: 14.2 with 4 slices (16.1 with 2, 17.0
// with 8); N 4096 K 4096: 11.1 with 8 (11.8 with 4); N 4096 K 12288: 20.9 with 8 (22.1 with 4); N 24576 and
// N 151936: one slice (34.4 and 188). With the norm kernel before it, time by time at 1 / 16 / 32 rows: 264 CTAs, N 4224 with 8
// slices against 4, K 2048 1.03 / 1.08 / 1.25, K 3072 0.96 / 1.00 / 0.84; 272 CTAs, N 4352 K 4096 1.29 at one row. 280 CTAs, N 8960
// with 4 slices against 2, K 1024 0.96 / 1.03 / 0.88, K 4096 0.93 / 0.89 / 0.82; 284 CTAs, N 9088 K 1024 0.97 / 1.32 / 0.93; 288 CTAs,
// N 9216 K 4096 1.36 / 1.30 / 1.23. Clusters of 2 all fit, but more than 256 CTAs of short slices do not pay for their sums: N 16512 with 2
// slices against one, K 2048 0.97 / 1.04 / 1.05, K 3072 0.91 / 0.98 / 0.96, K 8192 0.89 / 0.93 / 0.92; gated, where one tile's CTA
// would do all of the work behind them, they do: K 512 0.96 / 0.87 / 0.84.
int stream_slices(int N, int K, int glu) {
  const int tiles = (N + 127) / 128, num_kb = (K + 63) / 64;
  auto at_once = [&](int slices) {
    const int ctas = tiles * slices;
    if (ctas <= 256) return true;
    return slices == 4 ? ctas <= 280 : (slices == 2 && glu) || (num_kb >= 48 && (slices == 2 || ctas <= 264));
  };
  int c = 1;
  while (c < 8 && tiles * c < oi_sm_count() && num_kb / (2 * c) >= 2 && (t_streamed || at_once(2 * c))) c *= 2;
  if (g_opt[OI_OPT_FORCE_SLICES] > 0) c = g_opt[OI_OPT_FORCE_SLICES];
  while (c > 1 && (c - 1) * ((num_kb + c - 1) / c) >= num_kb) c /= 2;   // no slice may be left without a k block
  return c;
}

// Whether gemm_few.cu takes a decode product (us with the norm kernel before it, gemm_few.cu against the streaming kernel):
// * Rows of up to 3,072. Longer ones, which x's rows still fit, only where 148 CTAs take all of W at a time (N 2048 K 6144 6.9 against
//   9.1 at 8 rows): all of x has to reach every SM, and beside other long streams nothing is left of it (N 4096 K 4096 11.4 against
//   9.6 at 16 rows; Qwen3-8B sizes at 8 requests 68.2 against 68.4 ms).
// * Not the longest streams: N 32768 K 1024 15.0 against 14.3 at 16 rows, 13.3 against 13.6 at one.
// * A CTA spends some 0.65 us on a group of 16 rows however short they are, and as long on the last stage of a row as on a
//   full one. So the k that stages are too long for, over all groups of a CTA, are limited: K 64, 8 rows: N 6144 (2,880 of them)
//   3.4 against 3.5, N 12288 5.4 against 3.4, N 24576 9.4 against 3.5; K 512: N 12288 (3,072) 0.94 of the time, N 20480 1.22; K 1536:
//   N 12288 (3,072) 0.92, N 20480 1.09; K 2560: 0.95 and 1.05. K 1024 N 24576 (none) 0.88.
// * From nine rows on, x is twice as long. K 2,304 to 3,072: N 2288 (143 CTAs) 0.80 to 0.91 of the streaming kernel's time, N 2368 to
//   2880 1.03 to 1.13, N 3008 1.00, N 9728 0.87; K 2,112 0.93 at most. K 64 and 128: N 4736 1.0, N 5632 1.09 to 1.32, but gated (where the
//   streaming kernel has more to do behind its products) 0.70 to 0.87.
bool few_takes(const void* x, long long ldx, const void* W, long long ldw, int M, int N, int K, int glu) {
  if (t_streamed || g_opt[OI_OPT_FORCE_SLICES] != 0 || K < 64 || K % 64 || K > oi_gemm_few_max_k(M) || ldx % 16 || ldw % 8 ||
      (uintptr_t)x % 32 || (uintptr_t)W % 16)
    return false;
  const int groups = ((N + 15) / 16 + oi_sm_count() - 1) / oi_sm_count();      // of 16 rows, one CTA's
  const int spare = (1024 - K % 1024) % 1024 * groups;
  if (M > 8 && ((K > 2112 && N > 2288 && N < 3008) || (K < 256 && groups > 2 && !glu))) return false;
  return K <= 3072 ? N <= 24576 && spare <= 3072 : groups == 1 && (M <= 8 || N <= 2288);
}

// K slices of the mma.sync decode product, 0 if it does not take the shape (a slice's activations must fit in
// shared memory beside the 48 KB of weight rings). Four slices measured best for the short products.
int skinny_slices(int K) {
  auto fits = [&](int c) { return K % (32 * c) == 0 && 49152 + 32 * (K / c + 64) + 4096 <= 200 * 1024; };
  int chosen = 0;
  for (int c : {4, 2, 8, 1})
    if (fits(c)) {
      chosen = c;
      break;
    }
  const int forced = g_opt[OI_OPT_FORCE_SLICES];
  if (chosen && (forced == 1 || forced == 2 || forced == 4 || forced == 8) && fits(forced)) chosen = forced;
  return chosen;
}

int linear_bf16(void* out, int out_dtype, long long ldc, const void* x, long long ldx, const void* W, long long ldw, int M,
                int N, int K, void* stream) {
  const bool tma = tma_ok(x, ldx, W, ldw, K);
  if (g_opt[OI_OPT_BATCH_INVARIANT]) {
    // one kernel for every step shape: a row's sums are formed in the same order whatever else is in the step
    OI_REQUIRE(tma, "linear: batch-invariant products need 16-byte aligned bfloat16 operands with K %% 8 == 0");
    return oi_gemm_tcgen05(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, 256, OI_ACT_NONE, stream);
  }
  const int decode_gemm = g_opt[OI_OPT_DECODE_GEMM];
  if (M <= kDecodeMaxRows) {
    if (decode_gemm == 0 && tma)
      return oi_decode_product(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, 0, OI_ACT_NONE, 0.f, 0.f, stream);
    if (decode_gemm <= 1 && M <= kSkinnyMaxRows && tma && K >= 32) {
      const int c = skinny_slices(K);
      if (c) return oi_gemm_skinny(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, 0, 0, c, stream);
    }
  }
  if (M >= g_opt[OI_OPT_PAIR_MIN_ROWS] && g_opt[OI_OPT_PREFILL_GEMM] == 1 && tma)
    return oi_gemm_tcgen05_pair(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, OI_ACT_NONE, stream);
  if (oi_library_gemm_ready()) {
    if (oi_library_gemm(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, stream) == OI_OK) return OI_OK;
  }
  // without the vendor library (or for a shape it has no algorithm for): the hand-written kernels
  if (tma) {
    if (M >= g_opt[OI_OPT_PAIR_MIN_ROWS]) return oi_gemm_tcgen05_pair(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, OI_ACT_NONE, stream);
    return oi_gemm_tcgen05(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, 256, OI_ACT_NONE, stream);
  }
  return oi_gemm_generic(out, out_dtype, x, OI_BF16, W, OI_BF16, M, N, K, ldx, ldw, ldc, stream);
}

#define OI_TRY(expr)                  \
  do {                                \
    const int rc__ = (expr);          \
    if (rc__ != OI_OK) return rc__;   \
  } while (0)

}  // namespace

OI_API int oi_configure(int option, int value) {
  OI_REQUIRE(option >= 0 && option < OI_OPT_COUNT, "configure: unknown option %d", option);
  g_opt[option] = value;
  return OI_OK;
}

OI_API int oi_option(int option) { return option >= 0 && option < OI_OPT_COUNT ? g_opt[option] : -1; }

OI_API int oi_stream_slices(int N, int K) { return stream_slices(N, K, 0); }

OI_API int oi_streamed_products(int on) {
  const int was = t_streamed;
  t_streamed = on;
  return was;
}

OI_API int oi_decode_product(void* out, int out_dtype, long long ldc, const void* x, long long ldx, const void* W, long long ldw,
                             int M, int N, int K, int glu, int act, float p0, float p1, void* stream) {
  if (few_takes(x, ldx, W, ldw, M, N, K, glu)) return oi_gemm_few(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, glu, act, p0, p1, stream);
  const int c = stream_slices(N, K, glu);
  if (glu) return oi_gemm_stream_glu(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, c, act, p0, stream);
  if (act != OI_ACT_NONE) return oi_gemm_stream_unary(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, c, act, p0, p1, stream);
  return oi_gemm_stream(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, c, OI_ACT_NONE, stream);
}

OI_API int oi_linear(void* out, int out_dtype, long long ldc, const void* x, int x_dtype, long long ldx, const void* W,
                     int w_dtype, long long ldw, int M, int N, int K, void* stream) {
  OI_REQUIRE(M >= 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
  if (M == 0) return OI_OK;
  if (x_dtype == OI_BF16 && w_dtype == OI_BF16) return linear_bf16(out, out_dtype, ldc, x, ldx, W, ldw, M, N, K, stream);
  // anything with a float32 operand: float32 accumulation on the ordinary pipes, k ascending
  return oi_gemm_generic(out, out_dtype, x, x_dtype, W, w_dtype, M, N, K, ldx, ldw, ldc, stream);
}

namespace {
// 2: the tcgen05 product forms the activation in its epilogue; 1: the streaming product does; 0: nobody does
int gated_mlp_fusion(int dtype, int w_dtype, int M, int hidden, int inter, int act_block, const void* x, const void* w) {
  if (dtype != OI_BF16 || w_dtype != OI_BF16 || act_block != 64) return 0;
  const bool tma = tma_ok(x, hidden, w, hidden, hidden);
  if ((M >= kFusedMinRows || g_opt[OI_OPT_BATCH_INVARIANT]) && inter % 128 == 0) return tma ? 2 : 0;
  if (!g_opt[OI_OPT_BATCH_INVARIANT] && g_opt[OI_OPT_DECODE_GEMM] == 0 && M > 0 && M <= kDecodeMaxRows && tma &&
      (2 * inter) % 128 == 0)
    return 1;
  return 0;
}
}  // namespace

OI_API int oi_gated_mlp_needs_gate_up(int dtype, int w_dtype, int M, int hidden, int inter, int act_block) {
  // for 16-byte aligned operands, which is what this package's buffers and weights are
  return gated_mlp_fusion(dtype, w_dtype, M, hidden, inter, act_block, nullptr, nullptr) == 0 ? 1 : 0;
}

OI_API int oi_gated_mlp(void* out, const void* x, int dtype, int M, int hidden, int inter, const void* w_gate_up,
                        int w_dtype, const void* w_down, int w_down_dtype, int act, int act_block, void* act_buf,
                        void* gate_up_buf, void* stream) {
  OI_REQUIRE(M >= 0 && hidden > 0 && inter > 0, "gated_mlp: bad sizes M=%d hidden=%d inter=%d", M, hidden, inter);
  OI_REQUIRE(act == OI_ACT_SILU || act == OI_ACT_GELU_TANH, "gated_mlp: unknown activation code %d", act);
  OI_REQUIRE(act_block > 0 && inter % act_block == 0, "gated_mlp: block %d does not divide inter %d", act_block, inter);
  if (M == 0) return OI_OK;
  const int fusion = gated_mlp_fusion(dtype, w_dtype, M, hidden, inter, act_block, x, w_gate_up);
  if (fusion == 2) {
    // Short sums (K <= 2048) of fewer than 2,048 rows stay with single CTAs: a tile's products are then no longer than
    // its epilogue, which the pairs' larger tile does not hide, and there are too few of the larger tiles to go round.
    const bool pairs = M >= g_opt[OI_OPT_PAIR_MIN_ROWS] && (hidden > 2048 || M >= 2048);
    const int tile = g_opt[OI_OPT_BATCH_INVARIANT] ? 256 : (pairs ? kPair : 256);
    if (tile == kPair)
      OI_TRY(oi_gemm_tcgen05_pair(act_buf, OI_BF16, inter, x, hidden, w_gate_up, hidden, M, 2 * inter, hidden, act, stream));
    else
      OI_TRY(oi_gemm_tcgen05(act_buf, OI_BF16, inter, x, hidden, w_gate_up, hidden, M, 2 * inter, hidden, tile, act, stream));
  } else if (fusion == 1) {
    OI_TRY(oi_decode_product(act_buf, OI_BF16, inter, x, hidden, w_gate_up, hidden, M, 2 * inter, hidden, 1, act, 0.f, 0.f, stream));
  } else {
    OI_REQUIRE(gate_up_buf != nullptr, "gated_mlp: this shape needs the gate|up scratch buffer");
    OI_TRY(oi_linear(gate_up_buf, dtype, 2 * inter, x, dtype, hidden, w_gate_up, w_dtype, hidden, M, 2 * inter, hidden, stream));
    OI_TRY(oi_silu_mul(act_buf, gate_up_buf, dtype, M, inter, act_block, act, stream));
  }
  return oi_linear(out, dtype, hidden, act_buf, dtype, inter, w_down, w_down_dtype, inter, M, hidden, inter, stream);
}

OI_API int oi_dense_mlp(float* out, const void* x, int dtype, int M, int hidden, int inter, const void* w_up, int w_up_dtype,
                        const void* w_down, int w_down_dtype, const void* act_pq, int pq_dtype, float a_p, float a_n, void* z_buf,
                        void* stream) {
  OI_REQUIRE(M >= 0 && hidden > 0 && inter > 0, "dense_mlp: bad sizes M=%d hidden=%d inter=%d", M, hidden, inter);
  if (M == 0) return OI_OK;
  // the activation in the up-projection's epilogue where a hand-written product takes the shape, else on its own
  const bool fusable = dtype == OI_BF16 && w_up_dtype == OI_BF16 && tma_ok(x, hidden, w_up, hidden, hidden);
  if (fusable && !g_opt[OI_OPT_BATCH_INVARIANT] && M <= kDecodeMaxRows && g_opt[OI_OPT_DECODE_GEMM] == 0) {
    OI_TRY(oi_decode_product(z_buf, dtype, inter, x, hidden, w_up, hidden, M, inter, hidden, 0, OI_ACT_XIELU, a_p, a_n, stream));
  } else if (fusable && (M >= kFusedMinRows || g_opt[OI_OPT_BATCH_INVARIANT])) {   // 33..127 rows: the library's product is faster
    const int pairs = !g_opt[OI_OPT_BATCH_INVARIANT] && M >= g_opt[OI_OPT_PAIR_MIN_ROWS] && (hidden > 2048 || M >= 2048);
    OI_TRY(oi_gemm_tcgen05_unary(z_buf, dtype, inter, x, hidden, w_up, hidden, M, inter, hidden, pairs, OI_ACT_XIELU, a_p, a_n, stream));
  } else {
    OI_TRY(oi_linear(z_buf, dtype, inter, x, dtype, hidden, w_up, w_up_dtype, hidden, M, inter, hidden, stream));
    OI_TRY(oi_xielu(z_buf, z_buf, dtype, act_pq, pq_dtype, (long long)M * inter, stream));
  }
  return oi_linear(out, OI_F32, hidden, z_buf, dtype, inter, w_down, w_down_dtype, inter, M, hidden, inter, stream);
}

OI_API int oi_attention_layer(const OiAttnStep* s, const OiAttnLayer* l, void* stream) {
  OI_REQUIRE(s && l, "attention_layer: null description");
  const int tokens = s->tokens;
  if (tokens == 0) return OI_OK;
  const bool fused = l->rope_mode == 1 && s->tensor_core && s->fuse_rope && !l->interleaved;
  OI_REQUIRE(!(fused && (l->mods.sinks || l->mods.slopes || l->mods.softcap > 0.f || l->mods.qt_every > 0 || l->mods.keep_first > 0)),
             "attention_layer: a step with the rotation fused into the decode kernel cannot modify its scores");
  OI_REQUIRE(l->qkv && l->out && l->k_cache && l->v_cache && s->block_table && s->kv_lens && s->cu_seqlens,
             "attention_layer: a tensor of the step or of the layer is missing");
  OI_REQUIRE(l->rope_mode == 0 || ((!l->write_kv || s->slot_mapping) && (!l->cos_tab || s->positions)),
             "attention_layer: the rotation and the cache write need the step's positions and slots");
  OI_REQUIRE(s->tensor_core || (s->token_req && s->positions), "attention_layer: the general kernel needs token_req and positions");
  if (l->rope_mode == 1 && !fused)
    OI_TRY(oi_qk_norm_rope_kv(l->qkv, l->dtype, l->q_row_stride, tokens, l->nq, l->nkv, l->hd, l->q_norm_w, l->k_norm_w,
                              l->norm_dtype, l->eps, l->w_offset, l->cos_tab, l->sin_tab, l->cos_tab ? l->rot_half : 0,
                              l->cos_tab ? l->max_pos : 0, s->positions, s->slot_mapping, l->k_cache, l->v_cache,
                              s->page_stride, s->page_size, l->write_kv, l->interleaved, stream));
  if (!s->tensor_core)
    return oi_attention_generic(l->qkv, l->q_row_stride, l->out, l->out_row_stride, l->dtype, l->k_cache, l->v_cache,
                                s->page_stride, s->page_size, s->block_table, s->bt_stride, s->token_req, s->positions,
                                tokens, l->nq, l->nkv, l->hd, l->scale, l->window, &l->mods, stream);
  if (fused) {
    OI_REQUIRE(s->num_tile_items == 0 && s->num_decode_items > 0, "attention_layer: the fused rotation needs a step of single tokens");
    return oi_attention_decode_rope(l->qkv, l->q_row_stride, l->out, l->out_row_stride, l->k_cache, l->v_cache, s->page_stride,
                                    s->page_size, s->block_table, s->bt_stride, s->cu_seqlens, s->kv_lens, s->decode_items,
                                    s->num_decode_items, s->row_splits, tokens, l->nq, l->nkv, l->hd, l->scale, l->window,
                                    s->part_o, s->part_lse, s->max_splits, s->merge_in_kernel, l->q_norm_w, l->k_norm_w,
                                    l->norm_dtype, l->eps, l->w_offset, l->cos_tab, l->sin_tab, l->rot_half, l->max_pos,
                                    s->positions, s->slot_mapping, l->write_kv, stream);
  }
  const OiScoreMods* mods = (l->mods.sinks || l->mods.slopes || l->mods.softcap > 0.f || l->mods.qt_every > 0 || l->mods.keep_first > 0) ? &l->mods : nullptr;
  if (s->num_tile_items && s->use_tcgen05 && !mods)
    OI_TRY(oi_attention_tcgen05(l->qkv, l->q_row_stride, tokens, l->out, l->out_row_stride, l->k_cache, l->v_cache,
                                s->page_stride, s->page_size, s->num_pages, s->block_table, s->bt_stride, s->cu_seqlens,
                                s->kv_lens, s->tile_items, s->num_tile_items, l->nq, l->nkv, l->hd, l->scale, l->window,
                                s->row_splits, s->tile_split, s->part_o, s->part_lse, s->max_splits, stream));
  else if (s->num_tile_items)
    OI_TRY(oi_attention_mma_mods(l->qkv, l->q_row_stride, l->out, l->out_row_stride, l->k_cache, l->v_cache, s->page_stride,
                                 s->page_size, s->block_table, s->bt_stride, s->cu_seqlens, s->kv_lens, s->tile_items,
                                 s->num_tile_items, s->row_splits, tokens, s->tile_split, l->nq, l->nkv, l->hd, l->scale, l->window,
                                 s->part_o, s->part_lse, s->max_splits, s->rows_per_cta, mods, stream));
  if (s->num_decode_items)
    OI_TRY(oi_attention_decode_mods(l->qkv, l->q_row_stride, l->out, l->out_row_stride, l->k_cache, l->v_cache, s->page_stride,
                                    s->page_size, s->block_table, s->bt_stride, s->cu_seqlens, s->kv_lens, s->decode_items,
                                    s->num_decode_items, s->row_splits, tokens, l->nq, l->nkv, l->hd, l->scale, l->window,
                                    s->part_o, s->part_lse, s->max_splits, s->merge_in_kernel, mods, stream));
  return OI_OK;
}

namespace {
// A decode-sized step without norm kernels inside the layer stack: the products that end a residual branch (O, down)
// add the residual and leave the next norm's inputs behind, the products that follow (gate/up, QKV) scale their
// rows (gemm_stream.cu). Taken, when switched on (OI_OPT_FUSE_NORM, off by default), for up to 32 rows of a bfloat16
// model whose weights are all bfloat16 and TMA-readable.
// Measured on B200, it is no gain: 5 instead of 7 kernels per layer, but Qwen3-8B sizes at batch 8 run 3.56 ms a step
// against 3.50 ms with the norm kernels (batch 1: 3.22 against 3.19; Qwen3-0.6B sizes, batch 8: 1.19 against 1.11).
// The norm kernel's 2-3 us are not idle time: under it the product behind it, already resident, fills its ring of
// weight tiles, which it can only do once the product before has left the SMs; without the norm kernel that filling
// stands in the open, and the products that end a branch are 1-3 us longer for the residual's round trip through L2.
bool fused_norm_step(const OiModelDesc* m, const OiStepDesc* st) {
  if (!g_opt[OI_OPT_FUSE_NORM] || g_opt[OI_OPT_BATCH_INVARIANT] || g_opt[OI_OPT_DECODE_GEMM] != 0) return false;
  if (st->tokens > kDecodeMaxRows || m->dtype != OI_BF16 || !st->xs || !st->ssq || m->hidden % 8) return false;
  if (st->ssq_stride % 4 || st->ssq_stride < 8 * ((m->hidden + 127) / 128)) return false;
  for (int i = 0; i < m->num_layers; ++i) {
    const OiLayerDesc& L = m->layers[i];
    const int q_dim = L.attn.nq * L.attn.hd;
    if (L.w_qkv_dtype != OI_BF16 || L.w_o_dtype != OI_BF16 || L.w_gate_up_dtype != OI_BF16 || L.w_down_dtype != OI_BF16) return false;
    if (L.act_block != 64 || (2 * L.inter) % 128 || L.inter % 8 || q_dim % 8) return false;
    if ((uintptr_t)L.w_qkv % 16 || (uintptr_t)L.w_o % 16 || (uintptr_t)L.w_gate_up % 16 || (uintptr_t)L.w_down % 16) return false;
  }
  return true;
}

int forward_fused_norm(const OiModelDesc* m, const OiStepDesc* st, void* stream) {
  const int T = st->tokens, H = m->hidden;
  __nv_bfloat16* h = (__nv_bfloat16*)st->h;
  __nv_bfloat16* xs = (__nv_bfloat16*)st->xs;
  const float inv_width = 1.f / (float)H;
  int units = 0;   // partial sums of squares that the last residual product left per row
  for (int i = 0; i < m->num_layers; ++i) {
    const OiLayerDesc& L = m->layers[i];
    OI_REQUIRE(L.attn_step >= 0 && L.attn_step < st->num_attn_steps, "forward: layer %d names attention step %d of %d", i,
               L.attn_step, st->num_attn_steps);
    const int q_dim = L.attn.nq * L.attn.hd;
    // ---- input norm + QKV
    if (i == 0) {
      OI_TRY(oi_rmsnorm(st->x, st->h, nullptr, OI_BF16, L.input_norm_w, L.input_norm_dtype, nullptr, T, H, L.input_eps,
                        L.input_offset, stream));
      OI_TRY(oi_gemm_stream(st->qkv, OI_BF16, L.qkv_rows, st->x, H, L.w_qkv, H, T, L.qkv_rows, H, stream_slices(L.qkv_rows, H, 0),
                            OI_ACT_NONE, stream));
    } else {
      OiStreamEpilogue ep = {};
      ep.ssq_in = st->ssq, ep.ssq_units = units, ep.ssq_stride = st->ssq_stride, ep.inv_width = inv_width, ep.eps = L.input_eps;
      OI_TRY(oi_gemm_stream_fused(st->qkv, OI_BF16, L.qkv_rows, xs, H, L.w_qkv, H, T, L.qkv_rows, H,
                                  stream_slices(L.qkv_rows, H, 0), OI_ACT_NONE, &ep, stream));
    }
    // ---- attention
    OiAttnLayer a = L.attn;
    a.qkv = st->qkv, a.q_row_stride = L.qkv_rows, a.out = st->attn, a.out_row_stride = q_dim, a.dtype = OI_BF16;
    OI_TRY(oi_attention_layer(&st->attn_steps[L.attn_step], &a, stream));
    // ---- O + residual, and what the post norm needs
    {
      const int c = stream_slices(H, q_dim, 0);
      OiStreamEpilogue ep = {};
      ep.residual = h, ep.ld_residual = H, ep.norm_w = L.post_norm_w, ep.norm_w_bf16 = L.post_norm_dtype == OI_BF16;
      ep.w_offset = L.post_offset, ep.xs = xs, ep.ld_xs = H, ep.ssq_out = st->ssq, ep.ssq_stride = st->ssq_stride;
      OI_TRY(oi_gemm_stream_fused(h, OI_BF16, H, st->attn, q_dim, L.w_o, q_dim, T, H, q_dim, c, OI_ACT_NONE, &ep, stream));
      units = ((H + 127) / 128) * c;
    }
    // ---- post norm + gate/up with the activation
    {
      OiStreamEpilogue ep = {};
      ep.ssq_in = st->ssq, ep.ssq_units = units, ep.ssq_stride = st->ssq_stride, ep.inv_width = inv_width, ep.eps = L.post_eps;
      OI_TRY(oi_gemm_stream_fused(st->act, OI_BF16, L.inter, xs, H, L.w_gate_up, H, T, 2 * L.inter, H,
                                  stream_slices(2 * L.inter, H, 1), L.act, &ep, stream));
    }
    // ---- down + residual, and what the next layer's input norm needs (the last layer: only the residual)
    {
      const int c = stream_slices(H, L.inter, 0);
      OiStreamEpilogue ep = {};
      ep.residual = h, ep.ld_residual = H;
      if (i + 1 < m->num_layers) {
        const OiLayerDesc& next = m->layers[i + 1];
        ep.norm_w = next.input_norm_w, ep.norm_w_bf16 = next.input_norm_dtype == OI_BF16, ep.w_offset = next.input_offset;
        ep.xs = xs, ep.ld_xs = H, ep.ssq_out = st->ssq, ep.ssq_stride = st->ssq_stride;
      }
      OI_TRY(oi_gemm_stream_fused(h, OI_BF16, H, st->act, L.inter, L.w_down, L.inter, T, H, L.inter, c, OI_ACT_NONE, &ep, stream));
      units = ((H + 127) / 128) * c;
    }
  }
  return OI_OK;
}
}  // namespace

OI_API int oi_forward(const OiModelDesc* m, const OiStepDesc* st, void* stream) {
  OI_REQUIRE(m && st && m->layers && (st->num_attn_steps == 0 || st->attn_steps), "forward: null description");
  const int T = st->tokens, H = m->hidden, dt = m->dtype;
  OI_REQUIRE(T >= 0 && H > 0, "forward: bad sizes tokens=%d hidden=%d", T, H);
  if (T == 0) return OI_OK;
  OI_TRY(oi_embedding(st->h, dt, m->embedding, m->embedding_dtype, st->token_ids, T, H, m->vocab, stream));
  if (m->embedding_scale != 1.f) OI_TRY(oi_scale_cap(st->h, dt, (long long)T * H, m->embedding_scale, 0.f, stream));
  const void* pending = nullptr;   // the last branch output, added by the norm that reads the row next
  const bool fused = fused_norm_step(m, st);
  if (fused) OI_TRY(forward_fused_norm(m, st, stream));
  for (int i = 0; i < (fused ? 0 : m->num_layers); ++i) {
    const OiLayerDesc& L = m->layers[i];
    OI_REQUIRE(L.attn_step >= 0 && L.attn_step < st->num_attn_steps, "forward: layer %d names attention step %d of %d", i,
               L.attn_step, st->num_attn_steps);
    OI_TRY(oi_rmsnorm(st->x, st->h, pending, dt, L.input_norm_w, L.input_norm_dtype, nullptr, T, H, L.input_eps,
                      L.input_offset, stream));
    OI_TRY(oi_linear(st->qkv, dt, L.qkv_rows, st->x, dt, H, L.w_qkv, L.w_qkv_dtype, H, T, L.qkv_rows, H, stream));
    OiAttnLayer a = L.attn;
    const int q_dim = a.nq * a.hd;
    a.qkv = st->qkv;
    a.q_row_stride = L.qkv_rows;
    a.out = st->attn;
    a.out_row_stride = q_dim;
    a.dtype = dt;
    OI_TRY(oi_attention_layer(&st->attn_steps[L.attn_step], &a, stream));
    OI_TRY(oi_linear(st->branch_a, dt, H, st->attn, dt, q_dim, L.w_o, L.w_o_dtype, q_dim, T, H, q_dim, stream));
    OI_TRY(oi_rmsnorm(st->x, st->h, st->branch_a, dt, L.post_norm_w, L.post_norm_dtype, nullptr, T, H, L.post_eps,
                      L.post_offset, stream));
    OI_TRY(oi_gated_mlp(st->branch_m, st->x, dt, T, H, L.inter, L.w_gate_up, L.w_gate_up_dtype, L.w_down, L.w_down_dtype, L.act, L.act_block,
                        st->act, st->gate_up, stream));
    pending = st->branch_m;
  }
  if (st->num_want > 0) {
    OI_REQUIRE(st->want_rows && st->wanted && st->logits, "forward: wanted rows without buffers");
    OI_TRY(oi_rmsnorm(st->wanted, st->h, pending, dt, m->final_norm_w, m->final_norm_dtype, st->want_rows, st->num_want, H,
                      m->final_eps, m->final_offset, stream));
    OI_TRY(oi_linear(st->logits, OI_F32, m->vocab, st->wanted, dt, H, m->head, m->head_dtype, H, st->num_want, m->vocab, H, stream));
    if (m->logit_soft_cap > 0.f)
      OI_TRY(oi_scale_cap(st->logits, OI_F32, (long long)st->num_want * m->vocab, 1.f, m->logit_soft_cap, stream));
  }
  return OI_OK;
}

// The averages behind layer `layer` (whose own has `results` earlier terms) that its launch may add up terms for. Only those whose
// coefficients are as many as their turn asks for: the kernel reads `results` + 1 of each. One that is not so, and what lies
// behind it, is left out here and refused by oi_forward_branch when its turn comes.
OI_API int oi_depth_ahead_layers(const OiBranchLayerDesc* layers, int num_layers, int layer, int results, OiDepthAhead* ahead) {
  OI_REQUIRE(layers && ahead && layer >= 0 && layer < num_layers && results >= 0, "depth_ahead_layers: layer %d of %d", layer, num_layers);
  ahead->next = 0;
  int terms = results + 2;
  for (int q = layer + 1; q < num_layers && ahead->next < kDepthAhead; ++q) {
    if (!layers[q].depth_coef) continue;
    if (layers[q].depth_terms != terms++) break;
    ahead->coef[ahead->next] = layers[q].depth_coef;
    ahead->coef_dtype[ahead->next++] = layers[q].depth_dtype;
  }
  return OI_OK;
}

OI_API int oi_forward_branch(const OiBranchModelDesc* m, const OiBranchStepDesc* st, void* stream) {
  OI_REQUIRE(m && st && m->layers && (st->num_attn_steps == 0 || st->attn_steps), "forward_branch: null description");
  const int T = st->tokens, H = m->hidden, dt = m->dtype;
  OI_REQUIRE(T >= 0 && H > 0, "forward_branch: bad sizes tokens=%d hidden=%d", T, H);
  if (T == 0) return OI_OK;
  OI_REQUIRE(dt == OI_F32 || st->low, "forward_branch: a bfloat16 model needs the rounded copy of the stream");
  const long long hist_stride = (long long)T * H;
  OI_TRY(oi_embedding(st->h, OI_F32, m->embedding, m->embedding_dtype, st->token_ids, T, H, m->vocab, stream));
  if (m->embedding_scale != 1.f) OI_TRY(oi_scale_cap(st->h, OI_F32, (long long)T * H, m->embedding_scale, 0.f, stream));
  int results = 0;             // entries of the history so far
  if (st->hist) {
    OI_CHECK_CUDA(cudaMemcpyAsync(st->hist, st->h, sizeof(float) * (size_t)T * H, cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
    results = 1;
  }
  bool low_valid = false;      // `low` holds the stream as it stands
  // A layer's last branch joins the stream and the average over the history is formed. From the fourth result on, one average
  // in four also adds up what the next three need of the history so far (OiDepthAhead; before that they are as short as what is left).
  int ahead_from = 0, ahead_used = 0, ahead_have = 0;
  auto join_averaged = [&](int i, const void* norm_w, int norm_dtype, float eps, float offset) {
    const OiBranchLayerDesc& L = m->layers[i];
    OiDepthAhead d = {};
    const int left = ahead_used < ahead_have ? ahead_used++ : -1;
    if (st->ahead && oi_branch_ahead_ok(st->h, st->branch, norm_w, st->hist, st->ahead, st->low, H, results + kDepthAhead)) {
      if (left >= 0) {
        d.sum = st->ahead + left * hist_stride;
        d.from = ahead_from;
      } else if (results >= 4) {
        OI_TRY(oi_depth_ahead_layers(m->layers, m->num_layers, i, results, &d));
        d.out = st->ahead;
        d.stride = hist_stride;
        ahead_from = results, ahead_used = 0, ahead_have = d.next;
      }
    }
    return oi_branch_norm_add_ahead(st->h, st->branch, OI_F32, norm_w, norm_dtype, T, H, eps, offset, st->hist, hist_stride, results,
                                    L.depth_coef, L.depth_dtype, st->low, d.from || d.next ? &d : nullptr, stream);
  };
  for (int i = 0; i < m->num_layers; ++i) {
    const OiBranchLayerDesc& L = m->layers[i];
    OI_REQUIRE(L.attn_step >= 0 && L.attn_step < st->num_attn_steps, "forward_branch: layer %d names attention step %d of %d", i,
               L.attn_step, st->num_attn_steps);
    // ---- what the mixer reads
    const void* u = st->u;
    if (L.conv_w) {
      OI_TRY(oi_short_conv(st->u, dt, st->h, OI_F32, L.conv_w, L.conv_w_dtype, L.conv_state, L.conv_state_stride, st->cu_seqlens,
                           st->token_req, st->state_slots, st->state_phase, T, st->requests, H, L.taps, L.add_input, 1, stream));
    } else if (dt == OI_F32) {
      u = st->h;
    } else {
      OI_REQUIRE(low_valid, "forward_branch: layer %d has no filter and nothing has rounded the stream yet", i);
      u = st->low;
    }
    // ---- queries | latent | gate, the latent's norm and page write, attention over the latent, the gate, the output
    OI_TRY(oi_linear(st->proj, dt, L.in_cols, u, dt, H, L.w_in, L.w_in_dtype, H, T, L.in_cols, H, stream));
    const size_t esize = dt == OI_F32 ? 4 : 2;
    const OiAttnStep& as = st->attn_steps[L.attn_step];
    if (L.latent_norm_w)
      OI_TRY(oi_latent_store(L.pages, as.page_stride, as.page_size, L.row, (const char*)st->proj + esize * L.latent_off, L.in_cols, dt,
                             L.latent_norm_w, L.latent_norm_dtype, as.slot_mapping, T, L.rank, L.latent_eps, L.latent_offset, stream));
    OiAttnLayer a = {};
    a.qkv = st->proj, a.out = st->mixed, a.k_cache = L.pages, a.v_cache = L.pages;
    a.q_row_stride = L.in_cols, a.out_row_stride = L.heads * L.row, a.dtype = dt;
    a.nq = L.heads, a.nkv = 1, a.hd = L.row, a.window = L.window, a.scale = L.scale;
    a.write_kv = 0, a.rope_mode = 0;
    OI_TRY(oi_attention_layer(&as, &a, stream));
    if (L.has_gate)
      OI_TRY(oi_head_gate(st->mixed, L.heads * L.row, (const char*)st->proj + esize * L.gate_off, L.in_cols, dt, T, L.heads, L.row, stream));
    OI_TRY(oi_linear(st->branch, OI_F32, H, st->mixed, dt, L.heads * L.row, L.w_out, L.w_out_dtype, L.heads * L.row, T, H,
                     L.heads * L.row, stream));
    // ---- the branches join the stream; the layer's last one also forms the average
    const bool averaged = L.depth_coef != nullptr;
    OI_REQUIRE(!averaged || (st->hist && L.depth_terms == results + 1), "forward_branch: layer %d averages %d terms, %d exist", i,
               L.depth_terms, results + 1);
    const bool has_ff = L.w_up != nullptr;
    if (!has_ff && averaged) OI_TRY(join_averaged(i, L.mixer_norm_w, L.mixer_norm_dtype, L.mixer_eps, L.mixer_offset));
    else OI_TRY(oi_branch_norm_add(st->h, st->branch, OI_F32, L.mixer_norm_w, L.mixer_norm_dtype, T, H, L.mixer_eps, L.mixer_offset, nullptr,
                                   hist_stride, results, nullptr, OI_F32, st->low, stream));
    if (has_ff) {
      OI_TRY(oi_dense_mlp(st->branch, dt == OI_F32 ? (const void*)st->h : st->low, dt, T, H, L.inter, L.w_up, L.w_up_dtype, L.w_down,
                          L.w_down_dtype, L.act_pq, L.pq_dtype, L.act_a_p, L.act_a_n, st->z, stream));
      if (averaged) OI_TRY(join_averaged(i, L.ff_norm_w, L.ff_norm_dtype, L.ff_eps, L.ff_offset));
      else OI_TRY(oi_branch_norm_add(st->h, st->branch, OI_F32, L.ff_norm_w, L.ff_norm_dtype, T, H, L.ff_eps, L.ff_offset, nullptr, hist_stride,
                                     results, nullptr, OI_F32, st->low, stream));
    }
    if (averaged) ++results;
    low_valid = st->low != nullptr;
  }
  if (st->num_want > 0) {
    OI_REQUIRE(st->want_rows && st->wanted && st->logits, "forward_branch: wanted rows without buffers");
    OI_TRY(oi_rmsnorm_cast(st->wanted, dt, st->h, OI_F32, m->final_norm_w, m->final_norm_dtype, st->want_rows, st->num_want, H,
                           m->final_eps, m->final_offset, stream));
    OI_TRY(oi_linear(st->logits, OI_F32, m->vocab, st->wanted, dt, H, m->head, m->head_dtype, H, st->num_want, m->vocab, H, stream));
    if (m->logit_soft_cap > 0.f || m->logit_scale != 1.f)
      OI_TRY(oi_scale_cap(st->logits, OI_F32, (long long)st->num_want * m->vocab, m->logit_scale, m->logit_soft_cap, stream));
  }
  return OI_OK;
}
