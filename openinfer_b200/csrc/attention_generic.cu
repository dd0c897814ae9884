// Paged causal attention, general form: any head_dim that is a multiple of 8 (up to 512), any
// number of heads and groups, an optional window or chunks, float32 or bfloat16 storage; prompt portions
// and single decoded tokens alike. A block of eight warps per token and query head, or two heads of a kv head together.
//
// s[i,j] = (q_i . k_j) * scale for first_visible(pos_i) <= j <= pos_i (and j among the sequence's kept first keys),
// online softmax in float32,
// o_i = sum_j p[i,j] v_j; query head h reads kv head h / (nq / nkv)
// (pegainfer-kernels/csrc/shared/paged_attention.cu:439-567; pegainfer-kernels/src/ops/attention.rs:507).
// The keys of a request are visited in tiles of 32 from the first visible one, shared out among the warps whatever else is
// in the batch, so a row's result does not depend on how the batch was cut.
//
// What bounds it is latency: a lane's dot product is one chain over a key of its own (512 bytes at 128 float32 numbers), so
// the loads of up to sixteen 16-byte pieces (see kAhead) are in flight before their products, and a row's key tiles run side by side. One warp a row with
// one load in flight took 255 us a layer for 2 rows of 200 keys and 16 heads of float32, 152 us for a prompt of 355 rows; now
// 12.7 us and 79.8 us (B200).
//
// This is the kernel of the true 32-bit path and of every shape the tuned kernels refuse.
//
// Score modifiers (OiScoreMods, all optional): the score of a query at position p is multiplied by
// 1 + coef * ln(floor((p + 1) / every) + 1); then capped, s <- cap * tanh(s / cap); then slope_h * (i - j) is taken off;
// and the softmax's denominator gets one more term exp(sink_h), which has no key and no value (it enters as the state
// the online softmax starts from: maximum sink_h, sum 1, nothing accumulated).
#include <type_traits>

#include "common.cuh"
#include "oi_api.h"

#define ATTN_MAX_HD 512   // heads of more than 256 elements (a wide latent read as keys and values) get a second instance

template <typename T>
struct Vec16;  // 16 bytes of T
template <>
struct Vec16<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float* out) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  }
};
template <>
struct Vec16<bf16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void load(const bf16* p, float* out) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 f = __bfloat1622float2(h[k]);
      out[2 * k] = f.x; out[2 * k + 1] = f.y;
    }
  }
};

constexpr int kAttnWarps = 8;

// kHeads: query heads of one kv head that a block takes together (their keys and values are then fetched once)
template <typename T, int kMaxHd, int kHeads>
__global__ void __launch_bounds__(kAttnWarps * 32) attention_generic_kernel(
    const T* __restrict__ q, int q_row_stride, T* __restrict__ out, int out_row_stride,
    const T* __restrict__ k_cache, const T* __restrict__ v_cache, long long page_stride, int page_size,
    const int* __restrict__ block_table, int bt_stride, const int* __restrict__ token_req,
    const int* __restrict__ positions, int nq, int nkv, int hd, float scale, int window, OiScoreMods mods) {
  pdl_wait();    // no early trigger: waiting blocks of the next kernel would take the place of this one's
  constexpr int VN = Vec16<T>::N, kAccs = kMaxHd / 32;
  constexpr int kAhead = kMaxHd > 128 ? 8 : 16;           // pieces of a key, and
  constexpr int kKeys = kAccs > 8 ? 4 : 32 / kAccs;       // keys' values, that are in flight together
  __shared__ __align__(16) float q_sh[kHeads][kMaxHd];
  __shared__ float acc_sh[kAttnWarps][kHeads][kMaxHd];
  __shared__ float m_sh[kAttnWarps][kHeads], l_sh[kAttnWarps][kHeads];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int token = blockIdx.x, head = blockIdx.y * kHeads;
  const int req = token_req[token];
  if (req < 0) return;     // padding row: the whole block leaves
  const int pos = positions[token];
  const int kvh = head / (nq / nkv);
  const int* bt = block_table + (size_t)req * bt_stride;

  const T* qp = q + (size_t)token * q_row_stride + (size_t)head * hd;
  for (int d = threadIdx.x; d < kHeads * hd; d += kAttnWarps * 32) q_sh[d / hd][d % hd] = to_f32(qp[d]);
  __syncthreads();

  const int first = first_visible(pos, window);
  const size_t row_elems = (size_t)nkv * hd;
  float acc[kHeads][kAccs], m[kHeads], l[kHeads], slope[kHeads];
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
#pragma unroll
    for (int r = 0; r < kAccs; ++r) acc[h][r] = 0.f;
    m[h] = -INFINITY, l[h] = 0.f;
    if (mods.sinks && warp == 0) { m[h] = mods.sinks[head + h]; l[h] = 1.f; }
    slope[h] = mods.slopes ? mods.slopes[head + h] : 0.f;
  }
  if (mods.qt_every > 0) scale *= 1.f + mods.qt_coef * logf((float)((pos + 1) / mods.qt_every) + 1.f);
  const float cap = mods.softcap, inv_cap = cap > 0.f ? 1.f / cap : 0.f;

  // the keys a row sees: [first, pos], and with kept first keys also [0, min(keep_first, first)) behind the window
  const int kept_end = mods.keep_first > 0 ? min(mods.keep_first, first) : 0;
  const int kept_tiles = (kept_end + 31) / 32, tiles = kept_tiles + (pos + 1 - first + 31) / 32;
  for (int tile = warp; tile < tiles; tile += kAttnWarps) {
    const int base = tile < kept_tiles ? tile * 32 : first + (tile - kept_tiles) * 32;
    const int seg_hi = tile < kept_tiles ? kept_end : pos + 1;
    const int j = base + lane;
    float s[kHeads], p[kHeads];
#pragma unroll
    for (int h = 0; h < kHeads; ++h) s[h] = -INFINITY;
    long long at = 0;                      // where the lane's key lies in the cache (its value lies there in the other one)
    if (j < seg_hi) {
      at = (long long)bt[j / page_size] * page_stride + (long long)(j % page_size) * (long long)row_elems + (long long)kvh * hd;
      const T* kp = k_cache + at;
      float dot[kHeads];
#pragma unroll
      for (int h = 0; h < kHeads; ++h) dot[h] = 0.f;
      auto add_pieces = [&](int d, auto count) {
        constexpr int kCount = decltype(count)::value;
        float kv[kCount][VN];
#pragma unroll
        for (int u = 0; u < kCount; ++u) Vec16<T>::load(kp + d + u * VN, kv[u]);
#pragma unroll
        for (int u = 0; u < kCount; ++u)
#pragma unroll
          for (int e = 0; e < VN; ++e)
#pragma unroll
            for (int h = 0; h < kHeads; ++h) dot[h] += q_sh[h][d + u * VN + e] * kv[u][e];
      };
      constexpr int kCount = VN == 4 ? kAhead : kAhead / 2;
      int d = 0;
      for (; d + kCount * VN <= hd; d += kCount * VN) add_pieces(d, std::integral_constant<int, kCount>());
      for (; d < hd; d += VN) add_pieces(d, std::integral_constant<int, 1>());
#pragma unroll
      for (int h = 0; h < kHeads; ++h) {
        s[h] = dot[h] * scale;
        if (cap > 0.f) s[h] = cap * tanhf(s[h] * inv_cap);
        s[h] -= slope[h] * (float)(pos - j);
      }
    }
#pragma unroll
    for (int h = 0; h < kHeads; ++h) {
      const float m_new = fmaxf(m[h], warp_max(s[h]));
      const float m_ref = m_new == -INFINITY ? 0.f : m_new;      // a tile whose scores are all -inf weighs nothing
      p[h] = (j < seg_hi) ? expf(s[h] - m_ref) : 0.f;
      const float corr = expf(m[h] - m_ref);  // m = -inf on the first tile gives 0
      l[h] = l[h] * corr + warp_sum(p[h]);
#pragma unroll
      for (int r = 0; r < kAccs; ++r) acc[h][r] *= corr;
      m[h] = m_new;
    }
    const int n_valid = min(32, seg_hi - base);
    auto add_values = [&](int jj, auto count) {                // `count` keys: all their loads first
      constexpr int kCount = decltype(count)::value;
      float v[kCount][kAccs];
#pragma unroll
      for (int u = 0; u < kCount; ++u) {
        const T* vp = v_cache + __shfl_sync(0xffffffffu, at, jj + u);
#pragma unroll
        for (int r = 0; r < kAccs; ++r) v[u][r] = lane + 32 * r < hd ? to_f32(vp[lane + 32 * r]) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kCount; ++u)
#pragma unroll
        for (int h = 0; h < kHeads; ++h) {
          const float pj = __shfl_sync(0xffffffffu, p[h], jj + u);
#pragma unroll
          for (int r = 0; r < kAccs; ++r) acc[h][r] += pj * v[u][r];
        }
    };
    int jj = 0;
    for (; jj + kKeys <= n_valid; jj += kKeys) add_values(jj, std::integral_constant<int, kKeys>());
    for (; jj < n_valid; ++jj) add_values(jj, std::integral_constant<int, 1>());
  }
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
    if (lane == 0) { m_sh[warp][h] = m[h]; l_sh[warp][h] = l[h]; }
#pragma unroll
    for (int r = 0; r < kAccs; ++r) acc_sh[warp][h][lane + 32 * r] = acc[h][r];
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
    float top = m_sh[0][h];
#pragma unroll
    for (int w = 1; w < kAttnWarps; ++w) top = fmaxf(top, m_sh[w][h]);
    if (top == -INFINITY) top = 0.f;
    float share[kAttnWarps], total = 0.f;
#pragma unroll
    for (int w = 0; w < kAttnWarps; ++w) {
      share[w] = expf(m_sh[w][h] - top);
      total += l_sh[w][h] * share[w];
    }
    T* op = out + (size_t)token * out_row_stride + (size_t)(head + h) * hd;
    const float inv_l = 1.f / total;
    for (int d = threadIdx.x; d < hd; d += kAttnWarps * 32) {
      float o = 0.f;
#pragma unroll
      for (int w = 0; w < kAttnWarps; ++w) o += acc_sh[w][h][d] * share[w];
      op[d] = from_f32<T>(o * inv_l);
    }
  }
}

OI_API int oi_attention_generic(const void* q, int q_row_stride, void* out, int out_row_stride, int dtype,
                                const void* k_cache, const void* v_cache, long long page_stride,
                                int page_size, const int* block_table, int bt_stride,
                                const int* token_req, const int* positions, int tokens, int nq, int nkv,
                                int hd, float scale, int window, const OiScoreMods* mods_in, void* stream) {
  OI_REQUIRE(tokens >= 0 && nq > 0 && nkv > 0 && nq % nkv == 0, "attention: bad head counts nq=%d nkv=%d", nq, nkv);
  OI_REQUIRE(hd > 0 && hd % 8 == 0 && hd <= ATTN_MAX_HD,
             "attention: head_dim %d unsupported (multiples of 8 up to %d)", hd, ATTN_MAX_HD);
  OI_REQUIRE(q_row_stride % 8 == 0 && page_stride % 8 == 0, "attention: strides must be multiples of 8 elements");
  OI_REQUIRE(page_size > 0, "attention: page_size %d", page_size);
  if (tokens == 0) return OI_OK;
  OiScoreMods mods = {};
  if (mods_in) mods = *mods_in;
  cudaStream_t s = (cudaStream_t)stream;
#define OI_ATTN_GENERIC(T, MAXHD, HEADS)                                                                                   \
  oi_launch(attention_generic_kernel<T, MAXHD, HEADS>, dim3(tokens, nq / HEADS), kAttnWarps * 32, 0, s, (const T*)q,       \
            q_row_stride, (T*)out, out_row_stride, (const T*)k_cache, (const T*)v_cache, page_stride, page_size,           \
            block_table, bt_stride, token_req, positions, nq, nkv, hd, scale, window, mods)
#define OI_ATTN_SIZES(T)                                                          \
  do {                                                                            \
    if (hd <= 128 && (nq / nkv) % 2 == 0) OI_ATTN_GENERIC(T, 128, 2);             \
    else if (hd <= 128) OI_ATTN_GENERIC(T, 128, 1);                               \
    else if (hd <= 256) OI_ATTN_GENERIC(T, 256, 1);                               \
    else OI_ATTN_GENERIC(T, 512, 1);                                              \
  } while (0)
  OI_REQUIRE(dtype == OI_F32 || dtype == OI_BF16, "attention: unknown dtype code %d", dtype);
  if (dtype == OI_F32) OI_ATTN_SIZES(float);
  else OI_ATTN_SIZES(bf16);
#undef OI_ATTN_SIZES
#undef OI_ATTN_GENERIC
  OI_CHECK_LAUNCH();
  return OI_OK;
}
