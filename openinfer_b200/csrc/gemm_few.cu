// out[M, N] = x[M, K] * W[N, K]^T for at most 16 rows of x, bfloat16 operands, float32 sums: the products of a decode
// step of few requests, whose chain of dependent kernels is as much the bound as their weights are.
//
// One CTA per SM owns whole rows of W, so no sums cross CTAs and there is no cluster:
//   warp 8     copies the CTA's rows into shared memory (cp.async.bulk, one copy per row of a stage, counted on an
//              mbarrier), as many as the ring holds before the kernel ahead on the stream has finished: a layer's
//              projections of small models are then completely on the chip before x exists;
//   warps 0-7  share out K (64-wide blocks in turn). After the wait a warp reads ITS part of x straight into the
//              registers that mma.sync takes as operand B (tokens on the 8-column side), so x passes through no shared
//              memory and no second barrier; 16 rows of W are operand A. The k index inside a 64-wide block is permuted
//              alike for both operands, so 32 contiguous bytes of a row are a lane's fragments of four products, and a
//              lane's 32-byte load of x, four of which make a cache line, is its fragments of them too. The eight warps'
//              sums meet in shared memory and are added in warp order.
// What follows the wait is therefore one trip to L2 for x, the products out of shared memory, one barrier of the CTA
// and the store, where the streaming kernel (gemm_stream.cu) has a TMA copy of x, a tensor-memory round trip, deposits in
// other CTAs' shared memory and a cluster barrier. Every CTA reads all of x: each starts at another place of the row,
// because all at the same place is a queue in front of few L2 slices (one row of 1,024 / 3,072: 830 / 2,670 cycles for the
// loads, with 64-byte pieces and one starting place).
//
// Rows of a stage are 2,048 + 16 bytes apart: the eight lanes that a 128-bit shared load serves at once (two rows, four
// pieces 32 bytes apart) then hit different banks.
//
// Measured (us, a norm kernel and the product in turn inside a graph, other weights every time; the streaming kernel ->
// this one), 1 / 8 / 16 rows: N 4096 K 1024 5.1 -> 3.6 / 5.5 -> 4.3 / 6.1 -> 5.3; N 1024 K 3072 5.6 -> 3.8 / 6.0 -> 4.0 / 6.4 -> 4.8;
// N 9216 K 2048 10.7 -> 8.0 / 11.6 -> 8.1 / 12.7 -> 9.0; N 12288 K 2048 gated 12.9 -> 10.2 / 13.1 -> 10.2 / 13.6 -> 11.1; N 2048 K 6144
// 8.5 -> 6.3 / 9.1 -> 6.9 (the norm alone: 1.3 to 2.3; the weights at the copy rate: 0.33 us per million). What bounds it: the
// stream where the ring is shorter than a CTA's rows, else the chain above. The ring: with half of it, so that two CTAs fit on an
// SM, N 12288 K 2048 takes 12.6 and N 2048 K 6144 7.9. Refills by one of the eight warps instead of a ninth: N 24576 K 4096 44
// instead of 33. Rows of 12,288 in halves over a cluster of two: 25 against 19 in the streaming kernel.
#include "oi_api.h"
#include "tcgen05.cuh"

namespace {

constexpr int kWarps = 8;                       // that multiply; one more copies
constexpr int kThreads = (kWarps + 1) * 32;
constexpr int kChunkBlocks = 2;                 // 64-wide k blocks of a warp in a stage
constexpr int kChunkK = kChunkBlocks * kWarps * 64;   // 1,024 k of a row in a stage
constexpr int kRowBytes = kChunkK * 2 + 16;
constexpr int kPartBytes = 8192;
constexpr int kRingBytes = 12 * 8 * kRowBytes;  // at most 194 KB

__device__ int g_few_error = 0;                 // set when a bounded wait ran out

struct FewArgs {
  const bf16* x;
  const bf16* W;
  void* out;
  long long ldx, ldw, ldc;
  int M, N, K, groups, stages, act;
  float p0, p1;
};

__device__ __forceinline__ void mma_bf16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 lds128(unsigned addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
// 32 bytes of x, past L1: other SMs have just written them
__device__ __forceinline__ void load_x(uint4 (&v)[2], const bf16* p) {
  asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0].x), "=r"(v[0].y), "=r"(v[0].z), "=r"(v[0].w), "=r"(v[1].x), "=r"(v[1].y), "=r"(v[1].z), "=r"(v[1].w)
               : "l"(p) : "memory");
}
__device__ __forceinline__ void bulk_load(unsigned dst, const void* src, unsigned bytes, unsigned bar, unsigned long long policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;\n"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar), "l"(policy) : "memory");
}

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(kWarps * 32) : "memory"); }
// The wait's loop with its limit is out of line: nearly every wait ends at once, and what these kernels have not run yet
// comes from L2 instruction by instruction.
__device__ __noinline__ bool wait_longer(unsigned bar, unsigned parity, volatile int* abort_flag, int code) {
  return tc::mbar_wait(bar, parity, abort_flag, &g_few_error, code);
}
__device__ __forceinline__ bool wait(unsigned bar, unsigned parity, volatile int* abort_flag, int code) {
  return tc::mbar_try_wait(bar, parity) || wait_longer(bar, parity, abort_flag, code);
}

// NT: tokens / 8; G: groups of eight rows of W that a stage holds; B: 64-wide k blocks of a warp over the whole row.
// kGlu: W's rows come in blocks of 64 gate rows and their 64 up rows; a stage holds eight of each, out is [M, N / 2].
template <int NT, int G, int B, typename TOut, bool kGlu>
__global__ void __launch_bounds__(kThreads, (B * NT <= 6 ? 2 : 1))   // two kernels in a row fit an SM's registers
gemm_few_kernel(const __grid_constant__ FewArgs a) {
  pdl_trigger();
  static_assert(!kGlu || G == 2, "a stage of a gated product holds gate and up rows");
  static_assert(B % kChunkBlocks == 0, "whole stages");
  constexpr int kStageBytes = 8 * G * kRowBytes;
  constexpr int kHeld = 4 / (NT * G);                        // groups whose sums wait for one barrier
  constexpr int kTokens = 8 * NT, kRows = 8 * G;
  static_assert(kHeld * kWarps * kTokens * kRows * 4 <= kPartBytes, "sums of the groups held");
  extern __shared__ __align__(128) unsigned char smem[];
  float* part = reinterpret_cast<float*>(smem);              // [held][warp][rows][tokens]
  const unsigned ring = tc::smem_u32(smem) + kPartBytes;
  const unsigned bars = ring + a.stages * kStageBytes;       // full[stages], empty[stages]
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kPartBytes + a.stages * kStageBytes + 16 * a.stages);
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (a.stages + s); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = a.K / 64;                                   // 64-wide k blocks of a row
  const int chunks = (a.K + kChunkK - 1) / kChunkK;
  const int turn = blockIdx.x % chunks;                      // the stage of a row that this CTA begins with
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      tc::mbar_init(full_bar(s), 1);
      tc::mbar_init(empty_bar(s), kWarps);
    }
    *abort_flag = 0;
    tc::mbar_fence_init();
  }
  __syncthreads();

  if (warp == kWarps) {
    // ---- weights, ahead of everything else
    const unsigned long long once = tc::policy_evict_first();
    int slot = 0, round = 0;
    bool ok = true;
    for (int grp = blockIdx.x; grp < a.groups && ok; grp += gridDim.x) {
      const int n_lane = kGlu ? (grp >> 3) * 128 + (grp & 7) * 8 + (lane & 7) + (lane >> 3) * 64 : grp * kRows + lane;
      const int rows = kGlu ? 16 : (a.N - grp * kRows < kRows ? a.N - grp * kRows : kRows);
      for (int c = 0; c < chunks; ++c) {
        if (round > 0) ok = __all_sync(0xffffffffu, wait(empty_bar(slot), (unsigned)(round - 1) & 1, abort_flag, 1));
        if (!ok) break;
        const int k0 = (c + turn < chunks ? c + turn : c + turn - chunks) * kChunkK, len = a.K - k0 < kChunkK ? a.K - k0 : kChunkK;
        if (lane == 0) tc::mbar_expect_tx(full_bar(slot), (unsigned)(rows * len * 2));
        __syncwarp();
        if (lane < rows) bulk_load(ring + slot * kStageBytes + lane * kRowBytes, a.W + (size_t)n_lane * a.ldw + k0, (unsigned)(len * 2), full_bar(slot), once);
        if (++slot == a.stages) slot = 0, ++round;
      }
    }
  } else {
    // ---- x
    const int g = lane >> 2, c4 = lane & 3;
    const int swap = (blockIdx.x / chunks) & 1;                // the block of a stage that this CTA takes first
    auto block_of = [&](int i) {                               // the i-th 64-wide block of this warp
      const int c = i / kChunkBlocks + turn;
      return ((c < chunks ? c : c - chunks) * kChunkBlocks + ((i & 1) ^ swap)) * kWarps + warp;
    };
    const unsigned my_w = ring + g * kRowBytes + warp * 128 + c4 * 32;
    bool ok = wait(full_bar(0), 0, abort_flag, 2);   // weights: not waited for behind x
    pdl_wait();
    uint4 xr[B][NT][2];
#pragma unroll
    for (int i = 0; i < B; ++i) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int blk = block_of(i), m = g + 8 * t;
        xr[i][t][0] = xr[i][t][1] = make_uint4(0, 0, 0, 0);
        if (i / kChunkBlocks < chunks && blk < nb && m < a.M) load_x(xr[i][t], a.x + (size_t)m * a.ldx + blk * 64 + c4 * 16);
      }
    }

    // ---- products
    int slot = 0, phase = 0, held = 0, first = blockIdx.x;
    for (int grp = blockIdx.x; grp < a.groups; grp += gridDim.x) {
      float acc[NT][2][4] = {};
#pragma unroll
      for (int c = 0; c < B / kChunkBlocks; ++c) {
        if (c < chunks) {
          if (ok) ok = wait(full_bar(slot), phase, abort_flag, 2);
          const unsigned src = my_w + slot * kStageBytes;
#pragma unroll
          for (int j = 0; j < kChunkBlocks; ++j) {
            const int i = c * kChunkBlocks + j;
            if (block_of(i) < nb) {
              const unsigned at = src + (j ^ swap) * kWarps * 128;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint4 lo = lds128(at + h * 16), hi = G > 1 ? lds128(at + 8 * kRowBytes + h * 16) : make_uint4(0, 0, 0, 0);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                  mma_bf16(acc[t][0], lo.x, hi.x, lo.y, hi.y, xr[i][t][h].x, xr[i][t][h].y);
                  mma_bf16(acc[t][1], lo.z, hi.z, lo.w, hi.w, xr[i][t][h].z, xr[i][t][h].w);
                }
              }
            }
          }
          __syncwarp();
          if (lane == 0) tc::mbar_arrive(empty_bar(slot));
          if (++slot == a.stages) slot = 0, phase ^= 1;
        }
      }
      float* dst = part + (held * kWarps + warp) * (kRows * kTokens);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
#pragma unroll
        for (int q = 0; q < G; ++q)
          *reinterpret_cast<float2*>(dst + (q * 8 + g) * kTokens + t * 8 + c4 * 2) =
              make_float2(acc[t][0][2 * q] + acc[t][1][2 * q], acc[t][0][2 * q + 1] + acc[t][1][2 * q + 1]);
      }
      const bool last = grp + gridDim.x >= a.groups;
      if (++held == kHeld || last) {
        consumers_sync();
        // one sum of eight a thread: every divisor is a power of two
        constexpr int kCols = kGlu ? 8 : kRows, kEach = kTokens * kCols;
        for (int e = threadIdx.x; e < held * kEach; e += kWarps * 32) {
          const int f = e / kEach, m = e / kCols % kTokens, col = e % kCols;
          const int n = (first + f * gridDim.x) * kCols + col;
          if (m < a.M && (kGlu || n < a.N)) {
            const float* src = part + f * kWarps * (kRows * kTokens) + col * kTokens + m;
            float sum = 0.f, up = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
              sum += src[w * (kRows * kTokens)];
              if (kGlu) up += src[w * (kRows * kTokens) + 8 * kTokens];
            }
            if (kGlu) sum = glu_act<true>(sum, up, a.act, a.p0);
            else sum = unary_act<true>(sum, a.act, a.p0, a.p1);
            reinterpret_cast<TOut*>(a.out)[(size_t)m * a.ldc + n] = from_f32<TOut>(sum);
          }
        }
        held = 0;
        first = grp + gridDim.x;
        if (!last) consumers_sync();
      }
    }
  }
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0)
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);        // copies still landing in this CTA's shared memory
  __syncthreads();
}

template <int NT, int G, int B, typename TOut, bool kGlu>
int launch(const FewArgs& args, cudaStream_t s) {
  FewArgs a = args;
  auto kernel = gemm_few_kernel<NT, G, B, TOut, kGlu>;
  constexpr int kStageBytes = 8 * G * kRowBytes, kMost = kRingBytes / kStageBytes;
  static bool configured = false;
  if (!configured) {
    OI_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPartBytes + kMost * (kStageBytes + 16) + 16));
    configured = true;
  }
  a.groups = kGlu ? a.N / 16 : (a.N + 8 * G - 1) / (8 * G);
  const int sms = oi_sm_count(), grid = a.groups < sms ? a.groups : sms;
  const long long wanted = (long long)((a.groups + grid - 1) / grid) * ((a.K + kChunkK - 1) / kChunkK);
  a.stages = wanted < kMost ? (int)wanted : kMost;
  oi_launch(kernel, dim3(grid), dim3(kThreads), kPartBytes + a.stages * (kStageBytes + 16) + 16, s, a);
  OI_CHECK_LAUNCH();
  return OI_OK;
}

template <int NT, int B, typename TOut>
int pick_rows(const FewArgs& a, bool glu, cudaStream_t s) {
  if (glu) return launch<NT, 2, B, TOut, true>(a, s);
  // Sixteen rows of W at a time: a group costs a barrier and a store whatever it holds (8 rows of x, N 12288 K 1024: 5.8 us, 7.1 with
  // groups of eight although these spread more evenly, 88 rows a CTA instead of 96; N 24576 K 3072 25.4 and 32.0; at 16 rows of x short
  // rows of W would rather have three groups of eight than two of sixteen, N 3720 K 128 3.75 and 3.96). Eight where every
  // CTA has one group: at 16 rows of x N 1024 K 512 0.60 and 0.67 of the streaming kernel's time, K 1024 0.65 and 0.76 (up to eight rows
  // would rather have sixteen there too, 3.0 and 2.8 us, but a row's sums must not depend on how many rows there are).
  return a.N <= 8 * oi_sm_count() ? launch<NT, 1, B, TOut, false>(a, s) : launch<NT, 2, B, TOut, false>(a, s);
}

template <int NT, typename TOut>
int pick_k(const FewArgs& a, bool glu, cudaStream_t s) {
  const int chunks = (a.K + kChunkK - 1) / kChunkK;
  if (chunks <= 1) return pick_rows<NT, 2, TOut>(a, glu, s);
  if (chunks <= 2) return pick_rows<NT, 4, TOut>(a, glu, s);
  if (chunks <= 3) return pick_rows<NT, 6, TOut>(a, glu, s);
  if constexpr (NT == 1) {
    if (chunks <= 4) return pick_rows<NT, 8, TOut>(a, glu, s);
    return pick_rows<NT, 12, TOut>(a, glu, s);
  } else {
    return pick_rows<NT, 8, TOut>(a, glu, s);
  }
}

}  // namespace

// The longest row of W beside M rows of x (which lie in registers); 0: not this kernel's rows.
OI_API int oi_gemm_few_max_k(int M) { return M < 1 || M > 16 ? 0 : M <= 8 ? 6144 : 4096; }

// x: [M, K] bfloat16 (row stride ldx), W: [N, K] bfloat16 (row stride ldw), out: [M, N] bfloat16 or float32 (row stride
// ldc), 1 <= M <= 16, K a multiple of 64 up to oi_gemm_few_max_k(M); rows of x 32-byte aligned (base and stride), those of
// W 16-byte aligned. glu != 0: act is a gated activation's code, W's rows come in blocks of 64 gate rows and their 64 up
// rows (N a multiple of 128) and out is [M, N / 2]; p0 is its limit. Else act is OI_ACT_NONE or OI_ACT_XIELU with p0, p1.
OI_API int oi_gemm_few(void* out, int out_dtype, long long ldc, const void* x, long long ldx, const void* W, long long ldw, int M,
                       int N, int K, int glu, int act, float p0, float p1, void* stream) {
  OI_REQUIRE(M >= 1 && M <= 16 && N >= 1, "gemm_few: bad sizes M=%d N=%d", M, N);
  OI_REQUIRE(K >= 64 && K % 64 == 0 && K <= oi_gemm_few_max_k(M), "gemm_few: K=%d for %d rows", K, M);
  OI_REQUIRE(ldx % 16 == 0 && ldw % 8 == 0 && (uintptr_t)x % 32 == 0 && (uintptr_t)W % 16 == 0,
             "gemm_few: rows of x must be 32-byte aligned, those of W 16-byte aligned");
  OI_REQUIRE(out_dtype == OI_BF16 || out_dtype == OI_F32, "gemm_few: unknown output dtype code %d", out_dtype);
  OI_REQUIRE(glu ? (act == OI_ACT_SILU || act == OI_ACT_GELU_TANH || act == OI_ACT_SWIGLU_CLAMP) : (act == OI_ACT_NONE || act == OI_ACT_XIELU),
             "gemm_few: unknown activation code %d", act);
  OI_REQUIRE(!glu || N % 128 == 0, "gemm_few: a gated activation needs N %% 128 == 0 (N=%d)", N);
  FewArgs a = {};
  a.x = (const bf16*)x, a.W = (const bf16*)W, a.out = out, a.ldx = ldx, a.ldw = ldw, a.ldc = ldc;
  a.M = M, a.N = N, a.K = K, a.act = act, a.p0 = p0, a.p1 = p1;
  cudaStream_t s = (cudaStream_t)stream;
  if (M <= 8) return out_dtype == OI_BF16 ? pick_k<1, bf16>(a, glu != 0, s) : pick_k<1, float>(a, glu != 0, s);
  return out_dtype == OI_BF16 ? pick_k<2, bf16>(a, glu != 0, s) : pick_k<2, float>(a, glu != 0, s);
}

// 0 when no bounded wait has run out since the last call, else which role gave up (1 copies, 2 products). Synchronises.
OI_API int oi_gemm_few_status(int* status) {
  int v = 0;
  OI_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_few_error, sizeof(int)));
  if (v != 0) {
    int zero = 0;
    OI_CHECK_CUDA(cudaMemcpyToSymbol(g_few_error, &zero, sizeof(int)));
  }
  *status = v;
  return OI_OK;
}
