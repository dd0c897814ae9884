// The two products of routed experts for steps of few rows (up to 64 (row, choice) pairs), as a weight stream through the
// 5th-generation tensor cores: the form of gemm_stream.cu, with the weight rows of the experts that the step's pairs chose.
//
// The product is formed transposed: 128 weight rows of one expert are the M side of tcgen05.mma, ALL rows of the step its N
// side (padded to 16, 32 or 64 by TMA's zero fill), and only the columns of rows that chose the expert are stored. What the other
// columns cost is tensor-core time, of which a weight stream has plenty; in return nothing has to be sorted or gathered, and an
// expert's weights are read once however many rows chose it.
//
// Grid (c, tiles, experts): a cluster of c CTAs shares one tile of 128 weight rows (with the activation 64 gate rows and the
// 64 up rows of the same indices, two boxes of TMA; without it 128 neighbouring rows), CTA r of it streaming its share of the k
// blocks. Block z takes expert z, or, where experts outnumber pairs, the z-th expert in order of first choice; a cluster whose
// expert nobody chose leaves at once. Roles in a CTA (192 threads), as in gemm_stream.cu: warp 0 issues the TMA loads into a
// ring of stages, warp 1 the tensor-core products, warps 2-5 read the accumulator and deposit it with the CTA that adds up
// their rows' K slices (distributed shared memory, one cluster barrier, rank order). Every mbarrier wait is bounded. No load
// uses cluster multicast.
//
// Bound by the weights' bytes. Measured on B200 (us; a block per pair on the ordinary pipes before): see launch().
#include <cooperative_groups.h>

#include "oi_api.h"
#include "tcgen05.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kRowsPerTile = 128, kHalf = 64, BK = 64, kThreads = 192, kMaxPairs = 64;

__device__ int g_moe_stream_error = 0;     // set to a non-zero code when a bounded wait ran out

template <int BN>
struct Layout {
  static constexpr int kABytes = kRowsPerTile * BK * 2, kBBytes = BN * BK * 2, kStageBytes = kABytes + kBBytes;
  static constexpr int kRecvBytes = BN * kRowsPerTile * 4;           // partial sums [K slice][row of the step][rows of this CTA's share]
  static constexpr int kStages = (112 * 1024 - kRecvBytes) / kStageBytes;      // two CTAs fit on an SM
  static constexpr int kRecvOffset = kStages * kStageBytes;
  static constexpr int kBarOffset = kRecvOffset + kRecvBytes;        // full[kStages], empty[kStages], acc_full
  static constexpr int kNumBars = 2 * kStages + 1;
  static constexpr int kTotal = kBarOffset + kNumBars * 8 + 16;
  static constexpr int kTmemCols = BN < 32 ? 32 : BN;
  static_assert(kStages >= 3, "the ring keeps a load, a product and a spare in flight");
};

// out[p, col] for the pairs p that chose the block's expert; the product's row m of x belongs to pair p = m * top + j.
template <int BN, typename TOut, bool kGlu>
__global__ void __launch_bounds__(kThreads)
moe_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, TOut* __restrict__ out,
                  long long ld_out, int rows, int top, const int* __restrict__ ids, int pairs, int E, int N, int num_kb, int kb_per_rank,
                  float limit, int act) {
  pdl_trigger();
  using L = Layout<BN>;
  constexpr int kStages = L::kStages;
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ int pair_of[kMaxPairs];           // row of the step -> its pair that chose this expert, or -1
  __shared__ int s_expert;
  const unsigned smem_base = tc::smem_u32(smem);
  const bool misaligned = (smem_base & 1023u) != 0;   // the swizzled tiles need a 1024-byte aligned base (never seen otherwise)
  const unsigned bar_base = smem_base + L::kBarOffset;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  const unsigned acc_full = bar_base + 8u * (2 * kStages);
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(smem + L::kBarOffset + L::kNumBars * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* recv = reinterpret_cast<float*>(smem + L::kRecvOffset);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = blockIdx.x, csize = gridDim.x;
  constexpr int kOutRows = kGlu ? kHalf : kRowsPerTile;        // output columns per tile
  const int n0 = blockIdx.y * kOutRows;
  const int kb0 = rank * kb_per_rank;
  int nkb = num_kb - kb0;
  nkb = nkb < kb_per_rank ? nkb : kb_per_rank;
  nkb = nkb > 0 && !misaligned ? nkb : 0;
  if (misaligned && threadIdx.x == 0) atomicCAS(&g_moe_stream_error, 0, 9);

  if (threadIdx.x == 32) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(full_bar(s), 1);
      tc::mbar_init(empty_bar(s), 1);
    }
    tc::mbar_init(acc_full, 1);
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  if (warp == 1) {
    __syncwarp();
    tc::tmem_alloc(tc::smem_u32(tmem_slot), L::kTmemCols);
    tc::tmem_relinquish();
  }
  if (threadIdx.x >= 64 && threadIdx.x < 64 + kMaxPairs) pair_of[threadIdx.x - 64] = -1;
  pdl_wait();                                  // the choices, and x, are written by kernels before this one
  int id[2] = {-1, -1};                        // warp 0: the choices of pairs lane, lane + 32 (one behind the experts counts as none)
  if (warp == 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (lane + 32 * h < pairs) id[h] = ids[lane + 32 * h];
      if (id[h] >= E) id[h] = -1;
    }
    int e = blockIdx.z;
    if (gridDim.z < (unsigned)E) {
      bool again = false;
      for (int i = 0; i < 32; ++i) again |= __shfl_sync(0xffffffffu, id[0], i) == id[1];
      const unsigned same0 = __match_any_sync(0xffffffffu, id[0]), same1 = __match_any_sync(0xffffffffu, id[1]);
      const bool first0 = id[0] >= 0 && __ffs(same0) - 1 == lane, first1 = id[1] >= 0 && !again && __ffs(same1) - 1 == lane;
      const unsigned f0 = __ballot_sync(0xffffffffu, first0), f1 = __ballot_sync(0xffffffffu, first1), below = (1u << lane) - 1;
      const bool here0 = first0 && __popc(f0 & below) == e, here1 = first1 && __popc(f0) + __popc(f1 & below) == e;
      const unsigned who = __ballot_sync(0xffffffffu, here0 || here1);
      const int found = __shfl_sync(0xffffffffu, here0 ? id[0] : id[1], who ? __ffs(who) - 1 : 0);
      e = who ? found : -1;
    }
    const bool chosen = e >= 0 && __any_sync(0xffffffffu, id[0] == e || id[1] == e);
    if (lane == 0) s_expert = chosen ? e : -1;
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const int expert = s_expert;
  const unsigned tmem_base = *tmem_slot;
  if (expert < 0) {                            // nobody chose it: all CTAs of the cluster leave here
    if (warp == 1) tc::tmem_dealloc(tmem_base, L::kTmemCols);
    return;
  }
  if (csize > 1) tc::cluster_arrive();         // phase 0: "this CTA runs"; waited for before anyone writes into it

  if (warp == 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (id[h] == expert) pair_of[(lane + 32 * h) / top] = lane + 32 * h;
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      const unsigned long long once = tc::policy_evict_first();
      const int w0 = expert * (kGlu ? 2 * N : N) + n0, w1 = w0 + (kGlu ? N : kHalf);     // the tile's two halves
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % kStages;
        if (kb >= kStages && !tc::mbar_wait(empty_bar(s), (unsigned)((kb / kStages) - 1) & 1, abort_flag, &g_moe_stream_error, 1)) break;
        tc::mbar_expect_tx(full_bar(s), L::kStageBytes);
        const unsigned dst = smem_base + s * L::kStageBytes;
        tc::tma_load_2d_hint(dst, &map_w, (kb0 + kb) * BK, w0, full_bar(s), once);
        tc::tma_load_2d_hint(dst + kHalf * BK * 2, &map_w, (kb0 + kb) * BK, w1, full_bar(s), once);
        tc::tma_load_2d(dst + L::kABytes, &map_x, (kb0 + kb) * BK, 0, full_bar(s));
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      constexpr unsigned idesc = tc::idesc_bf16_f32(kRowsPerTile, BN);
      bool ok = true;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % kStages;
        ok = tc::mbar_wait(full_bar(s), (unsigned)(kb / kStages) & 1, abort_flag, &g_moe_stream_error, 2);
        if (!ok) break;
        tc::fence_after();
        const unsigned a_addr = smem_base + s * L::kStageBytes;
        const unsigned long long da = tc::desc_k_major_sw128(a_addr), db = tc::desc_k_major_sw128(a_addr + L::kABytes);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) tc::umma_bf16(tmem_base, da + 2ull * k, db + 2ull * k, idesc, (kb | k) != 0 ? 1u : 0u);
        tc::umma_commit(empty_bar(s));
      }
      if (ok && nkb > 0) tc::umma_commit(acc_full);
    }
  } else {
    // ------------------------------------------------------------------ accumulator read-out (warps 2..5)
    const int quarter = warp & 3, row = quarter * 32 + lane;      // weight row of this thread within the tile
    bool ok = true;
    if (nkb > 0) {
      ok = tc::mbar_wait(acc_full, 0, abort_flag, &g_moe_stream_error, 3);
      tc::fence_after();
    }
    if (csize > 1) tc::cluster_wait();                            // phase 0: every CTA of the cluster runs
    // Rows are shared out evenly: CTA j adds up rows [j * 128 / c, ...) (with the activation: gate rows [j * 64 / c, ...)
    // and, behind them in its buffer, the up rows of the same indices).
    const int share = kRowsPerTile / csize;
    int owner, local;
    if (kGlu) {
      const int idx = row & (kHalf - 1), per = kHalf / csize;
      owner = idx / per;
      local = (row >= kHalf ? per : 0) + idx % per;
    } else {
      owner = row / share;
      local = row % share;
    }
    float* const at = csize > 1 ? cg::this_cluster().map_shared_rank(recv, owner) : recv;
    const unsigned tmem_row = tmem_base + ((unsigned)(quarter * 32) << 16);
#pragma unroll 1
    for (int c0 = 0; c0 < BN && c0 < rows; c0 += 16) {
      unsigned v[16];
      if (nkb > 0 && ok) {
        tc::tmem_ld16(tmem_row + (unsigned)c0, v);
        tc::tmem_ld_wait();
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0u;
      }
      float* dst = at + (size_t)(rank * BN + c0) * share + local;
#pragma unroll
      for (int e = 0; e < 16; ++e) dst[e * share] = __uint_as_float(v[e]);
    }
  }

  // ------------------------------------------------------------------ sum over the K slices, teardown
  tc::fence_before();
  if (csize > 1) {
    if (warp < 2) tc::cluster_wait();     // the read-out warps waited before their first deposit
    tc::cluster_arrive();                 // phase 1: this CTA's deposits are made ...
    tc::cluster_wait();                   // ... and so are everybody's; nothing remote is touched after this
  } else {
    __syncthreads();
  }
  const int share = kRowsPerTile / csize, mine = kOutRows / csize, first = n0 + rank * mine;
  for (int i = threadIdx.x; i < rows * mine; i += kThreads) {
    const int m = i / mine, l = i - m * mine, p = pair_of[m];
    if (p < 0 || first + l >= N) continue;
    float sum = 0.f, up = 0.f;
    for (int q = 0; q < csize; ++q) {     // slice order: the result does not depend on timing
      const float* part = recv + (size_t)(q * BN + m) * share + l;
      sum += part[0];
      if (kGlu) up += part[mine];
    }
    out[(size_t)p * ld_out + first + l] = from_f32<TOut>(kGlu ? glu_act<false>(sum, up, act, limit) : sum);
  }
  if (*abort_flag && threadIdx.x == 0) {
    // copies that were issued may still be landing in this CTA's shared memory: give them time
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc(tmem_base, L::kTmemCols);
  }
}

template <int BN, typename TOut, bool kGlu>
int launch(void* out, long long ld_out, const void* x, long long ldx, int rows, int top, const void* w, int E, int N, int K, int act,
           float limit, const int* ids, int pairs, cudaStream_t s) {
  using L = Layout<BN>;
  CUtensorMap mw, mx;
  int rc = tc::make_map_2d_bf16(&mw, w, (long long)E * (kGlu ? 2 * N : N), K, K, kHalf);
  OI_REQUIRE(rc == 0, "moe_stream: tensor map for the weights failed (%d; -1: cuTensorMapEncodeTiled is not available)", rc);
  rc = tc::make_map_2d_bf16(&mx, x, rows, K, ldx, BN);
  OI_REQUIRE(rc == 0, "moe_stream: tensor map for x failed (%d)", rc);
  auto kernel = moe_stream_kernel<BN, TOut, kGlu>;
  static const cudaError_t allowed = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
  OI_CHECK_CUDA(allowed);
  // K slices: the fewest that give most SMs a CTA if every pair chose an expert of its own (which experts were chosen is not
  // known here), each slice at least four k blocks long; more only lengthen the sums over the slices. us for both products
  // inside a graph, 16 experts of 2,048 x 1,536, two a row: 1 row 24.2 / 19.0 / 17.3 / 22.6 with 1 / 2 / 4 / 8 slices, 2 rows
  // 25.8 / 24.2 / 26.8 / 36.9, 4 rows (7 experts) 31.5 / 36.5 / 43.8 / 63.5, 8 rows (10 experts, 189 MB) 39.5 / 48.0 / 55.4 / 88.3,
  // 16 rows 60.0 / 66.8 / 77.5 / 120; on the ordinary pipes with a block per pair 73, 96 and 96 for 4, 8 and 16 rows.
  constexpr int kOutRows = kGlu ? kHalf : kRowsPerTile;
  const int tiles = (N + kOutRows - 1) / kOutRows, experts = pairs < E ? pairs : E, num_kb = (K + BK - 1) / BK;
  int c = 1;
  while (c < 8 && (long long)tiles * experts * c < 128 && num_kb / (2 * c) >= 4) c *= 2;
  if (oi_option(OI_OPT_FORCE_SLICES) > 0) c = oi_option(OI_OPT_FORCE_SLICES);
  while (c > 1 && (c - 1) * ((num_kb + c - 1) / c) >= num_kb) c /= 2;      // no slice may be left without a k block
  oi_launch_cluster(kernel, dim3(c, tiles, experts), kThreads, L::kTotal, s, c, mw, mx, (TOut*)out, ld_out, rows, top, ids, pairs, E, N,
                    num_kb, (num_kb + c - 1) / c, limit, act);
  OI_CHECK_LAUNCH();
  return OI_OK;
}

}  // namespace

// out[p, :] (row stride ld_out) = W_e x[p / top] for every pair p < pairs = rows * top with e = ids[p] < E. x [rows, K] bfloat16,
// row stride ldx. act == OI_ACT_NONE: W [E, N, K], out float32; otherwise W [E, 2 N, K] (N gate rows, then N up rows) and
// out bfloat16 = the gated activation. A row's choices differ. K and ldx multiples of 8, 16-byte aligned operands.
OI_API int oi_moe_stream(void* out, long long ld_out, const void* x, long long ldx, int rows, int top, const void* w, int E, int N, int K,
                         int act, float limit, const int* ids, int pairs, void* stream) {
  OI_REQUIRE(rows >= 1 && top >= 1 && pairs == rows * top && pairs <= kMaxPairs, "moe_stream: %d rows of %d choices (at most %d pairs)", rows,
             top, kMaxPairs);
  OI_REQUIRE(E >= 1 && N >= 1 && K >= 8 && K % 8 == 0 && ldx % 8 == 0, "moe_stream: bad sizes E=%d N=%d K=%d", E, N, K);
  OI_REQUIRE((long long)E * 2 * N < (1LL << 31) && (N + kHalf - 1) / kHalf <= 65535, "moe_stream: %d experts of %d rows are too many", E, N);
  OI_REQUIRE((uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0, "moe_stream: operands must be 16-byte aligned");
  cudaStream_t s = (cudaStream_t)stream;
#define OI_MOE_STREAM(BN)                                                                                                       \
  return act == OI_ACT_NONE                                                                                                     \
             ? launch<BN, float, false>(out, ld_out, x, ldx, rows, top, w, E, N, K, act, limit, ids, pairs, s)                  \
             : launch<BN, bf16, true>(out, ld_out, x, ldx, rows, top, w, E, N, K, act, limit, ids, pairs, s)
  if (rows <= 16) OI_MOE_STREAM(16);
  if (rows <= 32) OI_MOE_STREAM(32);
  OI_MOE_STREAM(64);
#undef OI_MOE_STREAM
}

// 0 when no bounded wait has run out since the last call; otherwise which role gave up (1 producer, 2 MMA issuer, 3 read-out,
// 9: shared memory not aligned). Synchronises the device; clears the word.
OI_API int oi_moe_stream_status(int* status) {
  int v = 0;
  OI_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_moe_stream_error, sizeof(int)));
  if (v != 0) {
    int zero = 0;
    OI_CHECK_CUDA(cudaMemcpyToSymbol(g_moe_stream_error, &zero, sizeof(int)));
  }
  *status = v;
  return OI_OK;
}
