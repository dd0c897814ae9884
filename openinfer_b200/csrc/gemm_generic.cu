// C[M,N] = A[M,K] * W[N,K]^T with float32 accumulation on the ordinary (non-tensor) pipes.
//
// The product of the true 32-bit path (no reduced-precision matrix mode), and the fallback
// for operand types the tensor-core kernels do not take. Every output element is summed over k
// in ascending order in two levels: 256 consecutive products are added up in a register of their
// own, and that partial sum is then added to the total. The rounding error of a float32 sum grows
// with the size of the running total; with partial sums that start at zero every 256 terms it
// grows like sqrt(256) + sqrt(K / 256) instead of sqrt(K) (at K = 12,288: 23 against 111), which
// keeps a model of real width inside the tolerance that the tiny ones meet.
// Both kernels of this file form exactly these sums, so a row's result does not depend on M, on the
// other rows or on which kernel ran.
// Same contract as the reference's library call: row-major weight [out, in], no bias,
// float32 accumulate (pegainfer-kernels/csrc/shared/linear.cu:312-362).
//
// gemm_rows_kernel (few rows): a weight stream. The two-level sum lets the 256-term partial sums of one
// element be formed side by side: a warp takes 8 weight rows x 4 partial sums, one lane each, and fetches 128 bytes per
// lane and stage through its own cp.async ring (no block barrier before the end); the block's warps cover the rest of
// K, and the partial sums are added in order from shared memory. Bound by the weights' bytes, and below some 10 MB by latency.
// gemm_tile_kernel (more rows): 64 x 64 tiles, 8 x 4 sums a thread, the next tile's operands on their way in registers
// while this one is multiplied. Bound by the FMA pipe.
// Measured on B200 (us inside a graph, weights from memory; one kernel of 64 x 64 tiles, a load and a barrier per 16 terms
// before): 2 rows, N 4096 K 1024 7.7, N 1024 K 3072 5.9, all products of a Qwen3-0.6B layer 9.3 on average (140.7 before);
// 355 rows 93.8 on average (185.4 before). See the rule in launch() for where the line between the two lies.
#include "common.cuh"

namespace {
constexpr int kPartial = 256;           // terms per partial sum

__device__ __forceinline__ void cp_async_16(unsigned dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

// 16 bytes of T in shared memory as floats
__device__ __forceinline__ void unpack16(const float* p, float* o) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
}
__device__ __forceinline__ void unpack16(const bf16* p, float* o) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    o[2 * i] = f.x, o[2 * i + 1] = f.y;
  }
}

// ------------------------------------------------------------------------------------------------ few rows
// A stage of a warp: per partial sum (4 of them) and weight row (8) a segment of KS consecutive k, 128 bytes of W in a slot
// of 144 (so that the 16-byte reads of eight neighbouring lanes fall into different banks), and per partial sum and row of
// A the same KS terms.
template <typename TA, typename TW, int MG>
struct Rows {
  static constexpr int KS = 128 / (int)sizeof(TW);
  static constexpr int kSub = kPartial / KS;                       // stages per partial sum
  static constexpr int kWSlot = 144;
  static constexpr int kASeg = KS * (int)sizeof(TA), kASlot = kASeg + 16;
  static constexpr int kStage = 32 * kWSlot + 4 * MG * kASlot;
  static constexpr int kStages = 4;
  static constexpr int kWarp = kStages * kStage;
};

template <typename TA, typename TW, typename TC, int MG>
__global__ void gemm_rows_kernel(TC* __restrict__ C, const TA* __restrict__ A, const TW* __restrict__ W, int M, int N, int K,
                                 long long lda, long long ldw, long long ldc, int chunk_warps, int row_warps, int row_groups) {
  using L = Rows<TA, TW, MG>;
  constexpr int KS = L::KS, VW = 16 / (int)sizeof(TW), VA = 16 / (int)sizeof(TA), V = VW > VA ? VW : VA;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cw = warp % chunk_warps, rw = warp / chunk_warps;
  // the groups of rows of A that read the same weight rows are neighbours: the weights come from memory once
  const int n0 = ((int)blockIdx.x / row_groups * row_warps + rw) * 8, m0 = (int)blockIdx.x % row_groups * MG;
  const int chunks = (K + kPartial - 1) / kPartial;
  unsigned char* ring = smem + (size_t)warp * L::kWarp;
  float* parts = reinterpret_cast<float*>(smem + (size_t)(chunk_warps * row_warps) * L::kWarp) + (size_t)rw * chunks * 8 * MG;
  const unsigned ring_addr = (unsigned)__cvta_generic_to_shared(ring);
  const int row = lane & 7, part = lane >> 3;

  for (int c0 = cw * 4; c0 < chunks; c0 += chunk_warps * 4) {
    auto fetch_w = [&](int sub) {                  // the stage of terms [sub * KS, + KS) of the warp's four partial sums
      const unsigned base = ring_addr + (unsigned)(sub % L::kStages) * L::kStage;
#pragma unroll
      for (int i = 0; i < 8; ++i) {                // 32 segments x 8 pieces of 16 bytes: 8 lanes fetch one segment
        const int seg = i * 4 + (lane >> 3), piece = lane & 7;
        const int n = n0 + (seg & 7), k = (c0 + (seg >> 3)) * kPartial + sub * KS + piece * VW;
        const int left = (n < N && k < K) ? (K - k < VW ? K - k : VW) : 0;
        cp_async_16(base + seg * L::kWSlot + piece * 16, left ? W + (size_t)n * ldw + k : W, left * (int)sizeof(TW));
      }
    };
    auto fetch_a = [&](int sub) {
      const unsigned base = ring_addr + (unsigned)(sub % L::kStages) * L::kStage;
      constexpr int kPieces = L::kASeg / 16;
      for (int i = lane; i < 4 * MG * kPieces; i += 32) {
        const int seg = i / kPieces, piece = i % kPieces;
        const int m = m0 + seg % MG, k = (c0 + seg / MG) * kPartial + sub * KS + piece * VA;
        const int left = (m < M && k < K) ? (K - k < VA ? K - k : VA) : 0;
        cp_async_16(base + 32 * L::kWSlot + seg * L::kASlot + piece * 16, left ? A + (size_t)m * lda + k : A, left * (int)sizeof(TA));
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float sum[MG];
#pragma unroll
    for (int m = 0; m < MG; ++m) sum[m] = 0.f;
    __syncwarp();
    // the weights' first stages before the wait for the kernel that forms A (no kernel of a step writes weights): kSub >= 4
#pragma unroll
    for (int s = 0; s < L::kStages - 1; ++s) fetch_w(s);
    if (c0 == cw * 4) pdl_wait();
#pragma unroll
    for (int s = 0; s < L::kStages - 1; ++s) fetch_a(s);
    for (int sub = 0; sub < L::kSub; ++sub) {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(L::kStages - 2) : "memory");
      __syncwarp();                                                // everybody's pieces are there, and the stage before is read
      if (sub + L::kStages - 1 < L::kSub) fetch_w(sub + L::kStages - 1), fetch_a(sub + L::kStages - 1);
      else asm volatile("cp.async.commit_group;\n" ::: "memory");
      const unsigned char* st = ring + (size_t)(sub % L::kStages) * L::kStage;
      const TW* w = reinterpret_cast<const TW*>(st + lane * L::kWSlot);
      const unsigned char* a = st + 32 * L::kWSlot + part * MG * L::kASlot;
#pragma unroll
      for (int k = 0; k < KS; k += V) {
        float wv[V];
#pragma unroll
        for (int e = 0; e < V; e += VW) unpack16(w + k + e, wv + e);
#pragma unroll
        for (int m = 0; m < MG; ++m) {
          const TA* am = reinterpret_cast<const TA*>(a + m * L::kASlot) + k;
          float av[V];
#pragma unroll
          for (int e = 0; e < V; e += VA) unpack16(am + e, av + e);
#pragma unroll
          for (int e = 0; e < V; ++e) sum[m] = fmaf(av[e], wv[e], sum[m]);
        }
      }
    }
    if (c0 + part < chunks) {
#pragma unroll
      for (int m = 0; m < MG; ++m) parts[((size_t)(c0 + part) * 8 + row) * MG + m] = sum[m];
    }
  }
  pdl_trigger();     // not before: waiting blocks of the next kernel would take the place of this one's
  __syncthreads();
  for (int i = cw * 32 + lane; i < 8 * MG; i += chunk_warps * 32) {
    const int m = m0 + i / 8, n = n0 + i % 8;
    if (m >= M || n >= N) continue;
    float total = 0.f;
    for (int c = 0; c < chunks; ++c) total += parts[((size_t)c * 8 + i % 8) * MG + i / 8];
    C[(size_t)m * ldc + n] = from_f32<TC>(total);
  }
}

// ------------------------------------------------------------------------------------------------ many rows
constexpr int BM = 64, BN = 64, BK = 16, TM = 8, TN = 4;
constexpr int kGroup = (BM / TM) * (BN / TN);      // 128 threads form a tile's sums
constexpr int kGroupsMax = 4;
constexpr int kPitch = BM + 4;
constexpr int kGroupFloats = 2 * 2 * BK * kPitch;  // two buffers of both operands' tiles

// four consecutive k of a row, zero where the row or k ends; kVec: one aligned access (K % 4 == 0, so never past the end)
template <bool kVec>
__device__ __forceinline__ void load4(const float* p, int k, int K, bool row_ok, float* o) {
  if (kVec) {
    const float4 v = row_ok && k < K ? __ldg(reinterpret_cast<const float4*>(p + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
    o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = row_ok && k + e < K ? p[k + e] : 0.f;
  }
}
template <bool kVec>
__device__ __forceinline__ void load4(const bf16* p, int k, int K, bool row_ok, float* o) {
  if (kVec) {
    const uint2 v = row_ok && k < K ? __ldg(reinterpret_cast<const uint2*>(p + k)) : make_uint2(0u, 0u);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
    o[0] = lo.x, o[1] = lo.y, o[2] = hi.x, o[3] = hi.y;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = row_ok && k + e < K ? to_f32(p[k + e]) : 0.f;
  }
}

// A block of up to four groups of 128 threads. Group g forms the partial sums g, g + groups, ... of the tile; after every
// round the other groups leave theirs in shared memory and group 0 adds them up in order. Few tiles (a short prompt, a
// narrow product) then still give an SM sixteen warps: with one group a tile's loads were not hidden.
template <typename TA, typename TW, typename TC, bool kVec>
__global__ void __launch_bounds__(kGroup * kGroupsMax)
gemm_tile_kernel(TC* __restrict__ C, const TA* __restrict__ A, const TW* __restrict__ W, int M, int N, int K, long long lda,
                 long long ldw, long long ldc) {
  pdl_wait();    // no early trigger: waiting blocks of the next kernel would share the SMs with this product
  extern __shared__ __align__(16) float tile_smem[];
  const int groups = blockDim.x / kGroup, group = threadIdx.x / kGroup, tid = threadIdx.x % kGroup;
  float* own = tile_smem + (size_t)group * kGroupFloats;
  auto As = [&](int buf, int k) { return own + (buf * 2 * BK + k) * kPitch; };
  auto Ws = [&](int buf, int k) { return own + (buf * 2 * BK + BK + k) * kPitch; };
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[TM][TN], part[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  // a thread fetches 4 consecutive k of two rows of A and of W per tile
  const int lrow = tid / 4, lk = (tid % 4) * 4;
  float fa[2][4], fw[2][4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int am = m0 + lrow + 32 * h, wn = n0 + lrow + 32 * h;
      load4<kVec>(A + (size_t)(am < M ? am : 0) * lda, k0 + lk, K, am < M, fa[h]);
      load4<kVec>(W + (size_t)(wn < N ? wn : 0) * ldw, k0 + lk, K, wn < N, fw[h]);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        As(buf, lk + e)[lrow + 32 * h] = fa[h][e];
        Ws(buf, lk + e)[lrow + 32 * h] = fw[h][e];
      }
  };
  auto group_barrier = [&]() { asm volatile("bar.sync %0, %1;\n" ::"r"(group + 1), "n"(kGroup) : "memory"); };
  for (int round = 0; round < K; round += groups * kPartial) {
    const int first = round + group * kPartial, last = first + kPartial < K ? first + kPartial : K;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) part[i][j] = 0.f;
    if (first < K) {
      fetch(first);
      put(0);
      group_barrier();
      int buf = 0;
      for (int k0 = first; k0 < last; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < last;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
          float a[TM], w[TN];
#pragma unroll
          for (int i = 0; i < TM; i += 4) unpack16(As(buf, kk) + ty * TM + i, a + i);
          unpack16(Ws(buf, kk) + tx * TN, w);
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) part[i][j] = fmaf(a[i], w[j], part[i][j]);
        }
        if (more) put(buf ^ 1);      // last read before the previous tile's barrier
        group_barrier();
      }
    }
    if (group == 0) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] += part[i][j];
    }
    if (groups > 1) {                // the group's tiles are read: its partial sums take their place
      if (group > 0) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) own[(i * TN + j) * kGroup + tid] = part[i][j];
      }
      __syncthreads();
      if (group == 0) {
        for (int g = 1; g < groups && round + g * kPartial < K; ++g) {
          const float* theirs = tile_smem + (size_t)g * kGroupFloats;
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] += theirs[(i * TN + j) * kGroup + tid];
        }
      }
      if (round + groups * kPartial < K) __syncthreads();
    }
  }
  if (group > 0) return;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty * TM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * TN + j;
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(acc[i][j]);
    }
  }
}
static_assert(TM * TN * kGroup <= kGroupFloats, "a group's partial sums fit over its tiles");

bool aligned_rows(const void* p, long long ld, int esize, int bytes) { return (uintptr_t)p % bytes == 0 && (ld * esize) % bytes == 0; }

template <typename TA, typename TW, typename TC, int MG>
int launch_rows(void* C, const void* A, const void* W, int M, int N, int K, long long lda, long long ldw, long long ldc, cudaStream_t s) {
  using L = Rows<TA, TW, MG>;
  const int chunks = (K + kPartial - 1) / kPartial;
  // a warp per four partial sums, as many as fit into shared memory and eight at most (then each takes several runs of
  // four); where K is short and N long, several groups of eight weight rows share a block, which is then launched less often
  constexpr size_t kMaxSmem = 227 * 1024;
  const size_t parts = sizeof(float) * chunks * 8 * MG;
  int chunk_warps = (chunks + 3) / 4, row_warps = 1;
  while (chunk_warps > 1 && (chunk_warps > 8 || chunk_warps * (size_t)L::kWarp + parts > kMaxSmem)) --chunk_warps;
  while (row_warps * chunk_warps < 3 && (N + 15) / 16 / row_warps >= 4 * 148) row_warps *= 2;
  const size_t smem = row_warps * (chunk_warps * (size_t)L::kWarp + parts);
  const int row_groups = (M + MG - 1) / MG, blocks = (N + 8 * row_warps - 1) / (8 * row_warps);
  auto kernel = gemm_rows_kernel<TA, TW, TC, MG>;
  static const cudaError_t allowed = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem);
  OI_CHECK_CUDA(allowed);
  oi_launch(kernel, blocks * row_groups, 32 * chunk_warps * row_warps, smem, s, (TC*)C, (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldc,
            chunk_warps, row_warps, row_groups);
  OI_CHECK_LAUNCH();
  return OI_OK;
}

template <typename TA, typename TW, typename TC>
int launch(void* C, const void* A, const void* W, int M, int N, int K, long long lda, long long ldw,
           long long ldc, cudaStream_t s) {
  // The stream's time grows with groups of eight rows times N (2.0 ns a column and group at K = 1,024), that of a row of tiles not at
  // all up to 64 rows and with the waves of tiles beyond one an SM (30 us each at K = 1,024); both with K alike. us, stream /
  // tiles: N 4096, 3 groups K 1024 24 / 32, K 12288 346 / 353, 4 groups 32 / 32, 442 / 357; N 6144 K 4096 2 groups 112 / 120, 3 162 / 121;
  // N 12288 K 2048 2 groups 111 / 119, 3 161 / 119; N 24576 K 4096 1 group 214 / 351, 2 421 / 353; N 1024 K 3072 8 groups 47 / 93;
  // N 2048, 8 groups K 1024 32 / 33, K 2048 54 / 64.
  const long long groups_of_rows = (M + 7) / 8, waves = (N + 148 * BN - 1) / (148 * BN);
  const bool stream = M <= 64 && groups_of_rows * N < 15500 * waves;
  if (stream && K <= 32768 && aligned_rows(A, lda, sizeof(TA), 16) && aligned_rows(W, ldw, sizeof(TW), 16)) {
    if (M == 1) return launch_rows<TA, TW, TC, 1>(C, A, W, M, N, K, lda, ldw, ldc, s);
    if (M == 2) return launch_rows<TA, TW, TC, 2>(C, A, W, M, N, K, lda, ldw, ldc, s);
    if (M <= 4) return launch_rows<TA, TW, TC, 4>(C, A, W, M, N, K, lda, ldw, ldc, s);
    return launch_rows<TA, TW, TC, 8>(C, A, W, M, N, K, lda, ldw, ldc, s);
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  const bool vec = K % 4 == 0 && aligned_rows(A, lda, sizeof(TA), 4 * sizeof(TA)) && aligned_rows(W, ldw, sizeof(TW), 4 * sizeof(TW));
  auto kernel = vec ? gemm_tile_kernel<TA, TW, TC, true> : gemm_tile_kernel<TA, TW, TC, false>;
  // groups of threads per tile: as many as it takes to give the GPU four tiles' worth of warps per SM
  const long long tiles = (long long)grid.x * grid.y;
  int groups = 1;
  while (groups < kGroupsMax && tiles * groups * 2 <= 4 * 148 && groups * kPartial < K) groups *= 2;
  static const cudaError_t allowed = [] {
    const int most = kGroupsMax * kGroupFloats * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(gemm_tile_kernel<TA, TW, TC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(gemm_tile_kernel<TA, TW, TC, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
  }();
  OI_CHECK_CUDA(allowed);
  oi_launch(kernel, grid, kGroup * groups, groups * kGroupFloats * sizeof(float), s, (TC*)C, (const TA*)A, (const TW*)W, M, N, K, lda, ldw, ldc);
  OI_CHECK_LAUNCH();
  return OI_OK;
}
}  // namespace

// Leading dimensions are in elements; rows of A, W and C are contiguous in k / n.
OI_API int oi_gemm_generic(void* C, int c_dtype, const void* A, int a_dtype, const void* W, int w_dtype,
                           int M, int N, int K, long long lda, long long ldw, long long ldc, void* stream) {
  OI_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  OI_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm: leading dimension smaller than the row");
  if (M == 0) return OI_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int code = (a_dtype << 2) | (w_dtype << 1) | c_dtype;
  switch (code) {
    case 0b000: return launch<float, float, float>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b001: return launch<float, float, bf16>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b010: return launch<float, bf16, float>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b011: return launch<float, bf16, bf16>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b100: return launch<bf16, float, float>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b101: return launch<bf16, float, bf16>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b110: return launch<bf16, bf16, float>(C, A, W, M, N, K, lda, ldw, ldc, s);
    case 0b111: return launch<bf16, bf16, bf16>(C, A, W, M, N, K, lda, ldw, ldc, s);
  }
  OI_REQUIRE(false, "gemm: unknown dtype codes %d/%d/%d", a_dtype, w_dtype, c_dtype);
}
