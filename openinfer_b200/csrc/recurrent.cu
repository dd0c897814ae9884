// Recurrent mixers whose memory is a matrix per head: a scan over the rows of a step, request by request.
//
// Both kinds keep, per request and head, C [D keys x V values] in float32 and update it token by token:
//
//   kMatrixMemory (the mLSTM cell):  m' = max(f + m, i);  C' = e^(f + m - m') C + e^(i - m') k v^T;  n' likewise with k;
//                                    o = C'^T q / (max(|n' . q|, e^(-m')) + 1e-6);  i = cap tanh(zi / cap),
//                                    f = logsigmoid(cap tanh(zf / cap)); q arrives unscaled and is multiplied by q_scale
//   kGatedDelta (gated delta rule):  C <- diag(g) C;  d = beta (v - C^T k);  C <- C + k d^T;  o = C^T q, with k and q made
//                                    unit vectors (1e-6 inside the root), q times q_scale, beta = sigmoid(zb) and one decay
//                                    per key channel g = exp(-exp(A_h) softplus(a + dt))
//   kDeltaHeadDecay:                 the gated delta rule with one decay per head, g = exp(-exp(A_h) softplus(a_h + dt_h))
//   kLinearDecay (linear attention with one fixed decay per head, "lightning attention"):
//                                    C <- lambda_h C + k v^T;  o = C^T q, with q, k and v through silu first and no other scale
//
// Prompts and single decoded tokens take the same two launches. A first kernel forms, for all rows at once, what does
// not depend on earlier rows (gates, decays, unit vectors); then block (request, head, slice of value columns) walks the
// request's rows of the step in order, its slice of C in registers (a column's D numbers spread over 8 to 32 lanes), the
// rows' records staged in shared memory a chunk at a time (cp.async, two buffers), so that the loop over rows is the recurrence alone. The state
// lives in two copies that take turns ([slots][2][heads][elems], C stored column by column, then n and m): a step reads
// copy state_phase[request] and leaves the other, so no block reads what another writes. Everything is float32: the
// inputs are the float32 sums of the projections.
#include <type_traits>

#include "common.cuh"
#include "oi_api.h"

namespace {

enum : int { kMatrixMemory = 0, kGatedDelta = 1, kLinearDecay = 2, kDeltaHeadDecay = 3 };
constexpr int kThreads = 128;
constexpr int kMaxRegs = 16;   // key channels a thread holds of its column

struct ScanArgs {
  const float* qkv;            // [tokens, ld_qkv]: queries, keys (kv head major, D each) and values (head major, V each)
  long long ld_qkv;
  int q_off, k_off, v_off;
  const float* gates;          // [tokens, ld_gates]: matrix memory: zi at i_off + h, zf at f_off + h; delta: zb at i_off + h;
                               // delta with a decay per head: also a at f_off + h
  long long ld_gates;
  int i_off, f_off;
  const float* decay;          // delta: a [tokens, ld_decay], head major, D each
  long long ld_decay;
  const void* p0;              // matrix memory: bias of zi [H]; delta: dt [H * D] (a decay per head: [H]); linear decay: lambda [H]
  const void* p1;              // matrix memory: bias of zf [H]; delta: A [H]
  int p_dtype;
  float cap, q_scale;
  float* prep;                 // [tokens, H, rec]: what the scan reads per row and head (see the prepare kernels; the delta rule with a decay per channel: per run)
  int rec;
  float* state;
  long long state_stride;      // floats between slots (two copies inside)
  const int* cu_seqlens;
  const int* token_req;
  const int* state_slots;
  const int* state_phase;
  float* out;                  // [tokens, ld_out], head major, V each
  long long ld_out;
  int tokens, H, G, D, V;
};

// what a read-out is multiplied by for a gate's raw value z: sigmoid(z), or z sigmoid(z)
__device__ __forceinline__ float gate_value(float z, int act) {
  const float s = 1.f / (1.f + expf(-z));
  return act == OI_ACT_SILU ? z * s : s;
}
__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

// Everything of a row that does not depend on the rows before it, one warp per (row, head), so that the scan's loop is
// the recurrence alone. Record of rec >= 3 D + 2 floats: keys [D], queries [D], [D] that these modes leave unused, two scalars, padding.
//   matrix memory: keys as they are, queries times q_scale, the log gates i and f
//   linear decay:  silu of the keys, silu of the queries times q_scale; the head's values get their silu in place
template <int kMode>
__global__ void recurrent_prepare_kernel(ScanArgs a) {
  pdl_start();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= a.tokens * a.H) return;
  const int t = warp / a.H, h = warp - t * a.H, D = a.D;
  const int g = h / (a.H / a.G);
  const float* r = a.qkv + (size_t)t * a.ld_qkv;
  float* rec = a.prep + ((size_t)t * a.H + h) * a.rec;
  const float* gr = a.gates + (size_t)t * a.ld_gates;
  if (kMode == kLinearDecay) {
    for (int d = lane; d < D; d += 32) {
      const float k = r[a.k_off + g * D + d], q = r[a.q_off + g * D + d];
      rec[d] = k / (1.f + expf(-k));
      rec[D + d] = q / (1.f + expf(-q)) * a.q_scale;
    }
    float* v = const_cast<float*>(r) + a.v_off + (size_t)h * a.V;      // only this warp touches the head's values of the row
    for (int c = lane; c < a.V; c += 32) v[c] = v[c] / (1.f + expf(-v[c]));
  } else {
    for (int d = lane; d < D; d += 32) {
      rec[d] = r[a.k_off + g * D + d];
      rec[D + d] = r[a.q_off + g * D + d] * a.q_scale;
    }
    if (lane == 0) {
      const float zi = gr[a.i_off + h] + load_as_f32(a.p0, a.p_dtype, h), zf = gr[a.f_off + h] + load_as_f32(a.p1, a.p_dtype, h);
      const float fx = a.cap * tanhf(zf / a.cap);
      rec[3 * D] = a.cap * tanhf(zi / a.cap);
      rec[3 * D + 1] = fminf(fx, 0.f) - log1pf(expf(-fabsf(fx)));     // logsigmoid
    }
  }
}

// The records of the delta rule with one decay per head, by runs of four rows of a request (counted from its first row of the
// step). With P_i the product of the decays from the run's first row to row i, R_ij = g_i ... g_(j+1), and A the state in front
// of the run,
//   d_i = beta_i (v_i - P_i A^T k_i - sum_(j < i) R_ij (k_j . k_i) d_j),
//   o_i = P_i A^T q_i + sum_(j <= i) R_ij (k_j . q_i) d_j,        behind the run:  A <- P_3 A + sum_j R_3j k_j d_j,
// so everything a run needs of the state are eight dot products with A that do not wait for one another; what is left between
// its rows are numbers that no column of the state enters, and they are formed here. Record of row i: keys [D] (unit), queries
// [D] (unit, times q_scale), then, on a 16-byte boundary, beta, P_i, g_i, R_ij (k_j . k_i) for j = 0..2, R_ij (k_j . q_i) for j = 0..3 (zero for j > i),
// R_i(i-2), R_i(i-3). Records lie head by head, [H, tokens, rec].
constexpr int kDeltaScalars = 12;
__host__ __device__ constexpr int delta_scalars_at(int D) { return (2 * D + 3) & ~3; }      // on a 16-byte boundary, whatever D is

__global__ void delta_head_prepare_kernel(ScanArgs a) {
  pdl_start();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= a.tokens * a.H) return;
  const int t = warp / a.H, h = warp - t * a.H, D = a.D;
  const int g = h / (a.H / a.G);
  const int req = a.token_req[t];
  const int place = req >= 0 ? (t - a.cu_seqlens[req]) & 3 : 0;      // the row's place in its run
  const float* k_row = a.qkv + (size_t)t * a.ld_qkv + a.k_off + g * D;
  const float* q_row = a.qkv + (size_t)t * a.ld_qkv + a.q_off + g * D;
  float* rec = a.prep + ((size_t)h * a.tokens + t) * a.rec;
  float k2 = 0.f, q2 = 0.f, kq = 0.f, n2[3] = {0.f, 0.f, 0.f}, kk[3] = {0.f, 0.f, 0.f}, kqs[3] = {0.f, 0.f, 0.f};
  for (int d = lane; d < D; d += 32) {
    const float k = k_row[d], q = q_row[d];
    k2 += k * k, q2 += q * q, kq += k * q;
#pragma unroll
    for (int m = 0; m < 3; ++m)
      if (m < place) {
        const float b = k_row[d - (ptrdiff_t)(m + 1) * a.ld_qkv];
        n2[m] += b * b, kk[m] += b * k, kqs[m] += b * q;
      }
  }
  k2 = warp_sum(k2), q2 = warp_sum(q2), kq = warp_sum(kq);
#pragma unroll
  for (int m = 0; m < 3; ++m)
    if (m < place) n2[m] = warp_sum(n2[m]), kk[m] = warp_sum(kk[m]), kqs[m] = warp_sum(kqs[m]);
  const float kn = 1.f / sqrtf(k2 + 1e-6f), qn = a.q_scale / sqrtf(q2 + 1e-6f);
  for (int d = lane; d < D; d += 32) {
    rec[d] = k_row[d] * kn;
    rec[D + d] = q_row[d] * qn;
  }
  float decay = 1.f;                     // lane m: the decay of the row m rows up, of the same run
  if (lane <= place) {
    const float rate = expf(load_as_f32(a.p1, a.p_dtype, h));
    decay = expf(-rate * softplus_f(a.gates[(size_t)(t - lane) * a.ld_gates + a.f_off + h] + load_as_f32(a.p0, a.p_dtype, h)));
  }
  float R[4];                            // R[m]: the product over the row and the m rows above it
  R[0] = __shfl_sync(0xffffffffu, decay, 0);
#pragma unroll
  for (int m = 1; m < 4; ++m) R[m] = R[m - 1] * __shfl_sync(0xffffffffu, decay, m);     // (one beyond the run's first row)
  if (lane == 0) {
    float* s = rec + delta_scalars_at(D);
    s[0] = 1.f / (1.f + expf(-a.gates[(size_t)t * a.ld_gates + a.i_off + h]));
    s[1] = R[3];
    s[2] = R[0];
    float ck[3] = {0.f, 0.f, 0.f}, cq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j == place) cq[j] = kq * kn * qn;
#pragma unroll
      for (int m = 0; m < 3; ++m)        // the row m + 1 above this one is the run's row place - 1 - m
        if (place - 1 - m == j) {
          const float bn = R[m] / sqrtf(n2[m] + 1e-6f);
          cq[j] = kqs[m] * bn * qn;
          if (j < 3) ck[j] = kk[m] * bn * kn;
        }
    }
    s[3] = ck[0], s[4] = ck[1], s[5] = ck[2];
    s[6] = cq[0], s[7] = cq[1], s[8] = cq[2], s[9] = cq[3];
    s[10] = R[1], s[11] = R[2];
  }
}

// The records of the delta rule with a decay per key channel, by runs of up to four rows of a request (counted from its first row of
// the step; the last run may be shorter). With G(i, j) = g_(j+1) ... g_i channel by channel, and A the state in front of the run,
//   d_i = beta_i (v_i - A^T (G(i, -1) k_i) - sum_(j < i) ((G(i, j) k_j) . k_i) d_j),
//   o_i = A^T (G(i, -1) q_i) + sum_(j <= i) ((G(i, j) k_j) . q_i) d_j,
//   behind the run (of m rows):  A <- G(m-1, -1) A + sum_j (G(m-1, j) k_j) d_j.
// A run lies at its first row's place, ((head * tokens) + row) * rec: per row [beta, k_j . k_i for j = 0..2, k_j . q_i for j = 0..3 (both
// with their decays; zero beyond), G(i, -1) k_i, G(i, -1) q_i, G(m-1, i) k_i], then G(m-1, -1). Products of decays only: nothing
// is divided. One warp per (run, head).
constexpr int kRunScalars = 8;
__host__ __device__ constexpr int padded4(int D) { return (D + 3) & ~3; }
__host__ __device__ constexpr int run_row(int D) { return kRunScalars + 3 * padded4(D); }

// kPer: numbers of a row a lane keeps in registers (D at most 32 kPer), so that all of a run's loads are in flight at once. (Loads
// where they are used: 4 single rows, 8 heads of 128, 6.8 us, now 5.2; four requests of up to 1,500 rows 63 us, now 46.)
template <int kPer>
__global__ void __launch_bounds__(128) delta_channel_prepare_kernel(ScanArgs a) {
  pdl_trigger();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int t = warp / a.H, h = warp - t * a.H, D = a.D, D4 = padded4(D);
  const int req = t < a.tokens ? a.token_req[t] : -1;
  const bool live = req >= 0 && ((t - a.cu_seqlens[req]) & 3) == 0;
  const int m = live ? min(4, a.cu_seqlens[req + 1] - t) : 0;
  float rate = 0.f, dt[kPer];
  if (live) rate = expf(load_as_f32(a.p1, a.p_dtype, h));
#pragma unroll
  for (int c = 0; c < kPer; ++c) dt[c] = live && lane + 32 * c < D ? load_as_f32(a.p0, a.p_dtype, (size_t)h * D + lane + 32 * c) : 0.f;
  pdl_wait();       // (the step's metadata and the parameters before it)
  if (!live) return;
  const int g_head = h / (a.H / a.G);
  const float* k_row = a.qkv + (size_t)t * a.ld_qkv + a.k_off + g_head * D;
  const float* q_row = a.qkv + (size_t)t * a.ld_qkv + a.q_off + g_head * D;
  const float* a_row = a.decay + (size_t)t * a.ld_decay + (size_t)h * D;
  float* run = a.prep + ((size_t)h * a.tokens + t) * a.rec;
  float k[4][kPer], q[4][kPer], z[4][kPer], zb[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    zb[i] = i < m ? a.gates[(size_t)(t + i) * a.ld_gates + a.i_off + h] : 0.f;
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      const int d = lane + 32 * c;
      const bool in = i < m && d < D;
      k[i][c] = in ? k_row[(size_t)i * a.ld_qkv + d] : 0.f;
      q[i][c] = in ? q_row[(size_t)i * a.ld_qkv + d] : 0.f;
      z[i][c] = in ? a_row[(size_t)i * a.ld_decay + d] : 0.f;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i >= m) continue;
    float k2 = 0.f, q2 = 0.f;
#pragma unroll
    for (int c = 0; c < kPer; ++c) k2 += k[i][c] * k[i][c], q2 += q[i][c] * q[i][c];
    const float kn = 1.f / sqrtf(warp_sum(k2) + 1e-6f), qn = a.q_scale / sqrtf(warp_sum(q2) + 1e-6f);
#pragma unroll
    for (int c = 0; c < kPer; ++c) k[i][c] *= kn, q[i][c] *= qn;
  }
  float kk[4][3] = {}, kq[4][4] = {};
#pragma unroll
  for (int c = 0; c < kPer; ++c) {
    const int d = lane + 32 * c;
    if (d >= D) continue;
    float dec[4];            // dec[j]: k_j with the decays of the rows behind it, up to the current one
    float P = 1.f;               // G(i, -1)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i >= m) continue;
      const float g = expf(-rate * softplus_f(z[i][c] + dt[c]));
      P *= g;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < i) {
          dec[j] *= g;
          if (j < 3) kk[i][j] += dec[j] * k[i][c];
          kq[i][j] += dec[j] * q[i][c];
        }
      dec[i] = k[i][c];
      kq[i][i] += k[i][c] * q[i][c];
      run[(size_t)i * run_row(D) + kRunScalars + d] = P * k[i][c];
      run[(size_t)i * run_row(D) + kRunScalars + D4 + d] = P * q[i][c];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < m) run[(size_t)i * run_row(D) + kRunScalars + 2 * D4 + d] = dec[i];
    run[(size_t)m * run_row(D) + d] = P;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i >= m) continue;
    float s[kRunScalars];
    s[0] = 1.f / (1.f + expf(-zb[i]));
#pragma unroll
    for (int j = 0; j < 3; ++j) s[1 + j] = j < i ? warp_sum(kk[i][j]) : 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) s[4 + j] = j <= i ? warp_sum(kq[i][j]) : 0.f;
    if (lane < kRunScalars) {
      float v = s[0];
#pragma unroll
      for (int e = 1; e < kRunScalars; ++e) v = lane == e ? s[e] : v;
      run[(size_t)i * run_row(D) + lane] = v;
    }
  }
}

template <int kBytes>
__device__ __forceinline__ void cp_async(float* smem, const float* global) {
  const unsigned dst = (unsigned)__cvta_generic_to_shared(smem);
  if (kBytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(global) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(global) : "memory");
}

template <int kLanes>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Which key channel register i of lane j holds, and a row's D numbers into a thread's R registers. kVec4 (D a multiple of
// four): a lane holds runs of four neighbours, d = 4 (j + (i / 4) kLanes) + i % 4, and reads them 16 bytes at a time;
// otherwise d = j + i kLanes.
template <int kLanes, bool kVec4>
__device__ __forceinline__ int channel_of(int i, int j) {
  return kVec4 ? 4 * (j + (i >> 2) * kLanes) + (i & 3) : j + i * kLanes;
}
template <int kLanes, int R, bool kVec4>
__device__ __forceinline__ void load_channels(float (&dst)[R], const float* __restrict__ row, int D, int j) {
  if (kVec4) {
#pragma unroll
    for (int q = 0; q < R / 4; ++q) {
      const int d = 4 * (j + q * kLanes);
      const float4 v = d < D ? *reinterpret_cast<const float4*>(row + d) : make_float4(0.f, 0.f, 0.f, 0.f);
      dst[4 * q] = v.x, dst[4 * q + 1] = v.y, dst[4 * q + 2] = v.z, dst[4 * q + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int d = j + i * kLanes;
      dst[i] = d < D ? row[d] : 0.f;
    }
  }
}

// Block (request, head, slice of 2 kThreads / kLanes value columns): the request's rows of the step in order, up to four at a
// time, the slice of C in registers (the D numbers of two columns spread over kLanes lanes, R of each a lane), the rows' records
// staged in shared memory a chunk at a time. Two columns share what is read of a row, and the sums over the lanes of four rows
// are formed by halving. Bound by issue slots (0.75 instructions a clock of a scheduler with one warp). Four requests of up to
// 1,500 rows, 8 heads, with the records: matrix memory 1,131 -> 820 us with 128 keys and 256 values; linear attention, up to 2,000
// rows, 642 -> 468 us. (A lane's read-out in two sums instead of four takes 2 to 3 % less, and loses precision.)
template <int kMode, int kLanes, int R, bool kVec4>
__global__ void __launch_bounds__(kThreads) recurrent_scan_kernel(ScanArgs a, int chunk) {
  // (no early trigger: the blocks of the kernel behind this one would wait on the SMs this latency-bound loop needs)
  extern __shared__ __align__(16) float stage[];   // two buffers of [chunk][rec] records, then [chunk][cols] values
  constexpr bool kGates = kMode == kMatrixMemory;
  constexpr int kE = 2, kCols = kE * kThreads / kLanes;
  static_assert(kLanes >= 8, "a lane ends up with one column's and one row's sum");
  const int b = blockIdx.x, h = blockIdx.y;
  const int start = a.cu_seqlens[b], n_rows = a.cu_seqlens[b + 1] - start;
  if (n_rows <= 0 || a.token_req[start] < 0) {    // a padding request of a recorded step owns no state
    pdl_wait();
    return;
  }
  const int j = threadIdx.x % kLanes, pair = threadIdx.x / kLanes;
  const int c0 = blockIdx.z * kCols + kE * pair;
  const int D = a.D, V = a.V, rec = a.rec;
  const int elems = D * V + (kGates ? D + 1 : 0);
  const int phase = a.state_phase[b];
  const float* old = a.state + (size_t)a.state_slots[b] * a.state_stride + ((size_t)phase * a.H + h) * elems;
  float* fresh = a.state + (size_t)a.state_slots[b] * a.state_stride + ((size_t)(1 - phase) * a.H + h) * elems;
  pdl_wait();    // ahead of it the metadata alone: the old state may be what the kernel before leaves behind
  float C[kE][R], nn[R];
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int d = channel_of<kLanes, kVec4>(i, j);
#pragma unroll
    for (int e = 0; e < kE; ++e) C[e][i] = (c0 + e < V && d < D) ? old[(size_t)(c0 + e) * D + d] : 0.f;
    nn[i] = (kGates && d < D) ? old[(size_t)D * V + d] : 0.f;
  }
  if (kGates) m = old[(size_t)D * V + D];
  const float lam = kMode == kLinearDecay ? load_as_f32(a.p0, a.p_dtype, h) : 0.f;
  // which of four rows' sums this lane ends up with
  const int my_col = (j / (kLanes / 2)) & 1, my_row = ((j / (kLanes / 4)) & 1) * 2 + ((j / (kLanes / 8)) & 1);
  const bool writer = j % (kLanes / 8) == 0;

  // two buffers: the next chunk's records are on their way (cp.async) while this one is worked on
  const int buf_floats = chunk * (rec + kCols);
  auto request = [&](int t0, int buf) {
    const int n = min(chunk, n_rows - t0), rec4 = rec / 4;
    float* st = stage + (size_t)buf * buf_floats;
    float* vl = st + (size_t)chunk * rec;
    for (int i = threadIdx.x; i < n * rec4; i += kThreads) {
      const int tt = i / rec4, e = (i - tt * rec4) * 4;
      cp_async<16>(st + (size_t)tt * rec + e, a.prep + ((size_t)(start + t0 + tt) * a.H + h) * rec + e);
    }
    for (int i = threadIdx.x; i < n * kCols; i += kThreads) {
      const int tt = i / kCols, cc = blockIdx.z * kCols + (i - tt * kCols);
      if (cc < V) cp_async<4>(vl + i, a.qkv + (size_t)(start + t0 + tt) * a.ld_qkv + a.v_off + h * V + cc);
      else vl[i] = 0.f;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // Up to four rows at a time. The read-outs feed nothing, so the chain from row to row is one multiply-add a register (and
  // the gates' scalars), and the rows' sums over the lanes do not wait for one another: they are formed by halving, every
  // exchange leaving a lane half as many.
  auto walk = [&](const float* rows, const float* vals, int first_row, auto whole, int count) {
    constexpr bool kWhole = decltype(whole)::value;
    float num[4 * kE], den[4], low[4];       // sums [column][row]; denominators and their lower bounds [row]
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int e = 0; e < kE; ++e) num[e * 4 + u] = 0.f;
      den[u] = 0.f, low[u] = 1.f;
      if (!kWhole && u >= count) continue;
      const float* r = rows + (size_t)u * rec;
      float keep = lam, put = 1.f;
      if (kGates) {
        const float gi = r[3 * D], gf = r[3 * D + 1], m_new = fmaxf(gf + m, gi);
        keep = expf(gf + m - m_new), put = expf(gi - m_new);
        m = m_new;
        low[u] = expf(-m);
      }
      float k[R], q[R];
      load_channels<kLanes, R, kVec4>(k, r, D, j);
      load_channels<kLanes, R, kVec4>(q, r + D, D, j);
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        const float pv = kGates ? put * vals[u * kCols + kE * pair + e] : vals[u * kCols + kE * pair + e];
        float p[4] = {0.f, 0.f, 0.f, 0.f};       // four partial sums a lane: short chains of roundings
#pragma unroll
        for (int i = 0; i < R; ++i) {
          C[e][i] = fmaf(keep, C[e][i], k[i] * pv);
          p[i & 3] += C[e][i] * q[i];
        }
        num[e * 4 + u] = (p[0] + p[1]) + (p[2] + p[3]);
      }
      if (kGates) {
        float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < R; ++i) {
          nn[i] = fmaf(keep, nn[i], put * k[i]);
          p[i & 3] += nn[i] * q[i];
        }
        den[u] = (p[0] + p[1]) + (p[2] + p[3]);
      }
    }
#pragma unroll
    for (int half = 2 * kE, o = kLanes / 2; half > 0; half >>= 1, o >>= 1) {       // column, row, row
      const bool up = (j & o) != 0;
#pragma unroll
      for (int i = 0; i < 2 * kE; ++i)
        if (i < half) {
          const float send = up ? num[i] : num[i + half], kept = up ? num[i + half] : num[i];
          num[i] = kept + __shfl_xor_sync(0xffffffffu, send, o);
        }
      if (kGates && half == 2 * kE) {
#pragma unroll
        for (int u = 0; u < 4; ++u) den[u] += __shfl_xor_sync(0xffffffffu, den[u], o);
      } else if (kGates) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (i < half) {
            const float send = up ? den[i] : den[i + half], kept = up ? den[i + half] : den[i];
            den[i] = kept + __shfl_xor_sync(0xffffffffu, send, o);
          }
      }
    }
#pragma unroll
    for (int o = kLanes / 16; o > 0; o >>= 1) {
      num[0] += __shfl_xor_sync(0xffffffffu, num[0], o);
      if (kGates) den[0] += __shfl_xor_sync(0xffffffffu, den[0], o);
    }
    if (writer && c0 + my_col < V && (kWhole || my_row < count)) {
      const float bound = my_row < 2 ? (my_row == 0 ? low[0] : low[1]) : (my_row == 2 ? low[2] : low[3]);
      a.out[(size_t)(first_row + my_row) * a.ld_out + (size_t)h * V + c0 + my_col] = kGates ? num[0] / (fmaxf(fabsf(den[0]), bound) + 1e-6f) : num[0];
    }
  };
  request(0, 0);
  int turn = 0;
  for (int t0 = 0; t0 < n_rows; t0 += chunk, turn ^= 1) {      // chunk: a multiple of four
    const int n = min(chunk, n_rows - t0);
    if (t0 + chunk < n_rows) {
      request(t0 + chunk, turn ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float* stage_now = stage + (size_t)turn * buf_floats;
    const float* vals = stage_now + (size_t)chunk * rec;
    int tt = 0;
#pragma unroll 2
    for (; tt + 3 < n; tt += 4) walk(stage_now + (size_t)tt * rec, vals + tt * kCols, start + t0 + tt, std::true_type(), 4);
    if (tt < n) walk(stage_now + (size_t)tt * rec, vals + tt * kCols, start + t0 + tt, std::false_type(), n - tt);
    __syncthreads();                           // everyone has read this buffer before the chunk after next is requested into it
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int d = channel_of<kLanes, kVec4>(i, j);
    if (d >= D) continue;
#pragma unroll
    for (int e = 0; e < kE; ++e)
      if (c0 + e < V) fresh[(size_t)(c0 + e) * D + d] = C[e][i];
    if (kGates && blockIdx.z == 0 && pair == 0) fresh[(size_t)D * V + d] = nn[i];
  }
  if (kGates && blockIdx.z == 0 && threadIdx.x == 0) fresh[(size_t)D * V + D] = m;
}

// The scan of the delta rule with a decay per key channel: blocks and staging as above, a request's rows a run of up to four at a
// time (see delta_channel_prepare_kernel). kLanes lanes hold kE = 2 columns of the state, R numbers of each a lane, so that what a
// run brings is read from shared memory once for both; its sums over the lanes (two columns, four rows, key or query) are
// formed by halving, every exchange leaving a lane half as many. Bound by shared memory's and the shuffles' pipe: with a
// column a lane group and two rows at a time (eight trees of shuffles and 24 16-byte reads a pair and column group) four requests
// of up to 1,500 rows, 8 heads of 128 keys and values, took 788 us with the records, and this 435 us (with one chain of sums a
// lane instead of four 427 us).
template <int kLanes, int R, bool kVec4>
__global__ void __launch_bounds__(kThreads) delta_channel_scan_kernel(ScanArgs a, int chunk) {
  extern __shared__ __align__(16) float stage[];      // two buffers of [chunk / 4] runs, then [chunk][cols] values
  constexpr int kE = 2, kCols = kE * kThreads / kLanes;
  static_assert(kLanes >= 8, "a lane ends up with one column's and one row's sums");
  const int b = blockIdx.x, h = blockIdx.y;
  const int start = a.cu_seqlens[b], n_rows = a.cu_seqlens[b + 1] - start;
  if (n_rows <= 0 || a.token_req[start] < 0) {
    pdl_wait();
    return;
  }
  const int lane = threadIdx.x & 31, j = threadIdx.x % kLanes, pair = threadIdx.x / kLanes;
  const int c0 = blockIdx.z * kCols + kE * pair;
  const int D = a.D, V = a.V, D4 = padded4(D), row = run_row(D), full_run = 4 * row + D4;
  const int phase = a.state_phase[b];
  const float* old = a.state + (size_t)a.state_slots[b] * a.state_stride + ((size_t)phase * a.H + h) * D * V;
  float* fresh = a.state + (size_t)a.state_slots[b] * a.state_stride + ((size_t)(1 - phase) * a.H + h) * D * V;
  pdl_wait();    // ahead of it the metadata alone: the old state may be what the kernel before leaves behind
  float C[kE][R];
#pragma unroll
  for (int e = 0; e < kE; ++e)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int d = channel_of<kLanes, kVec4>(i, j);
      C[e][i] = (c0 + e < V && d < D) ? old[(size_t)(c0 + e) * D + d] : 0.f;
    }
  // which of a run's sums this lane ends up with, and which lane has row u's of column e
  const int my_col = (j / (kLanes / 2)) & 1, my_row = ((j / (kLanes / 4)) & 1) * 2 + ((j / (kLanes / 8)) & 1);
  const bool writer = j % (kLanes / 8) == 0;
  const int group = lane & ~(kLanes - 1);
  const int buf_floats = (chunk / 4) * full_run + chunk * kCols;
  auto request = [&](int t0, int buf) {
    const int n = min(chunk, n_rows - t0);
    float* st = stage + (size_t)buf * buf_floats;
    float* vl = st + (size_t)(chunk / 4) * full_run;
    for (int tt = 0; tt < n; tt += 4) {
      const int pieces = (min(4, n - tt) * row + D4) / 4;
      const float* src = a.prep + ((size_t)h * a.tokens + start + t0 + tt) * a.rec;
      float* dst = st + (size_t)(tt / 4) * full_run;
      for (int i = threadIdx.x; i < pieces; i += kThreads) cp_async<16>(dst + 4 * i, src + 4 * i);
    }
    for (int i = threadIdx.x; i < n * kCols; i += kThreads) {
      const int tt = i / kCols, cc = blockIdx.z * kCols + (i - tt * kCols);
      if (cc < V) cp_async<4>(vl + i, a.qkv + (size_t)(start + t0 + tt) * a.ld_qkv + a.v_off + h * V + cc);
      else vl[i] = 0.f;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // a run of m rows; the whole run has the loops without conditions
  auto walk = [&](const float* run, const float* vals, int first_row, auto whole, int m) {
    constexpr bool kWhole = decltype(whole)::value;
    float v[8 * kE];          // sums [column][row][key, query]
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float k[R], q[R];
      const bool live = kWhole || u < m;
      if (live) {
        load_channels<kLanes, R, kVec4>(k, run + (size_t)u * row + kRunScalars, D, j);
        load_channels<kLanes, R, kVec4>(q, run + (size_t)u * row + kRunScalars + D4, D, j);
      }
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        float pk[4] = {0.f, 0.f, 0.f, 0.f}, pq[4] = {0.f, 0.f, 0.f, 0.f};      // four partial sums a lane, as above
        if (live) {
#pragma unroll
          for (int i = 0; i < R; ++i) {
            pk[i & 3] += C[e][i] * k[i];
            pq[i & 3] += C[e][i] * q[i];
          }
        }
        v[(e * 4 + u) * 2] = (pk[0] + pk[1]) + (pk[2] + pk[3]);
        v[(e * 4 + u) * 2 + 1] = (pq[0] + pq[1]) + (pq[2] + pq[3]);
      }
    }
    float4 s0[4], s1;         // beta, k_0 . k, k_1 . k, k_2 . k of every row; k_0 . q .. k_3 . q of this lane's
    float want[kE][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool live = kWhole || u < m;
      s0[u] = live ? *reinterpret_cast<const float4*>(run + (size_t)u * row) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int e = 0; e < kE; ++e) want[e][u] = live ? vals[u * kCols + kE * pair + e] : 0.f;
    }
    s1 = kWhole || my_row < m ? *reinterpret_cast<const float4*>(run + (size_t)my_row * row + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int half = 4 * kE, o = kLanes / 2; half > 1; half >>= 1, o >>= 1) {       // column, row, row
      const bool up = (j & o) != 0;
#pragma unroll
      for (int i = 0; i < 4 * kE; ++i)
        if (i < half) {
          const float send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int o = kLanes / 16; o > 0; o >>= 1) {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      v[1] += __shfl_xor_sync(0xffffffffu, v[1], o);
    }
    float d[kE][4];
#pragma unroll
    for (int e = 0; e < kE; ++e) {
      float ak[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        ak[u] = __shfl_sync(0xffffffffu, v[0], group + e * (kLanes / 2) + (u >> 1) * (kLanes / 4) + (u & 1) * (kLanes / 8));
      d[e][0] = s0[0].x * (want[e][0] - ak[0]);
      d[e][1] = s0[1].x * (want[e][1] - ak[1] - s0[1].y * d[e][0]);
      d[e][2] = s0[2].x * (want[e][2] - ak[2] - s0[2].y * d[e][0] - s0[2].z * d[e][1]);
      d[e][3] = s0[3].x * (want[e][3] - ak[3] - s0[3].y * d[e][0] - s0[3].z * d[e][1] - s0[3].w * d[e][2]);
    }
    if (writer && c0 + my_col < V && (kWhole || my_row < m)) {
      const float d0 = my_col ? d[1][0] : d[0][0], d1 = my_col ? d[1][1] : d[0][1], d2 = my_col ? d[1][2] : d[0][2], d3 = my_col ? d[1][3] : d[0][3];
      a.out[(size_t)(first_row + my_row) * a.ld_out + (size_t)h * V + c0 + my_col] = v[1] + (s1.x * d0 + s1.y * d1) + (s1.z * d2 + s1.w * d3);
    }
    float G[R];
    load_channels<kLanes, R, kVec4>(G, run + (size_t)(kWhole ? 4 : m) * row, D, j);
#pragma unroll
    for (int e = 0; e < kE; ++e)
#pragma unroll
      for (int i = 0; i < R; ++i) C[e][i] *= G[i];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (!kWhole && u >= m) break;
      float k[R];
      load_channels<kLanes, R, kVec4>(k, run + (size_t)u * row + kRunScalars + 2 * D4, D, j);
#pragma unroll
      for (int e = 0; e < kE; ++e)
#pragma unroll
        for (int i = 0; i < R; ++i) C[e][i] += k[i] * d[e][u];
    }
  };
  request(0, 0);
  int turn = 0;
  for (int t0 = 0; t0 < n_rows; t0 += chunk, turn ^= 1) {      // chunk: a multiple of four, so that runs do not straddle it
    const int n = min(chunk, n_rows - t0);
    if (t0 + chunk < n_rows) {
      request(t0 + chunk, turn ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float* stage_now = stage + (size_t)turn * buf_floats;
    const float* vals = stage_now + (size_t)(chunk / 4) * full_run;
    int tt = 0;
#pragma unroll 2
    for (; tt + 3 < n; tt += 4) walk(stage_now + (size_t)(tt / 4) * full_run, vals + tt * kCols, start + t0 + tt, std::true_type(), 4);
    if (tt < n) walk(stage_now + (size_t)(tt / 4) * full_run, vals + tt * kCols, start + t0 + tt, std::false_type(), n - tt);
    __syncthreads();                           // everyone has read this buffer before the chunk after next is requested into it
  }
#pragma unroll
  for (int e = 0; e < kE; ++e)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int d = channel_of<kLanes, kVec4>(i, j);
      if (c0 + e < V && d < D) fresh[(size_t)(c0 + e) * D + d] = C[e][i];
    }
}

// The scan of the delta rule with one decay per head: blocks and staging as above, the request's rows four at a time (see
// delta_head_prepare_kernel), what is left over one at a time. kLanes lanes (16 or 32) hold two columns of the
// state, R numbers of each a lane, so that a row's key and query are read once for both. The sums of a run over the lanes (two
// columns, four rows, key or query) are formed by halving: every exchange leaves a lane half as many, until lane (column, row,
// kind) has its one.
template <int kLanes, int R, bool kVec4>
__global__ void __launch_bounds__(kThreads) delta_head_scan_kernel(ScanArgs a, int chunk) {
  extern __shared__ __align__(16) float stage[];
  constexpr int kE = 2;                             // columns a lane
  constexpr int kCols = kE * kThreads / kLanes, kRowStep = kLanes / (4 * kE), kKindStep = kLanes / (8 * kE);
  const int b = blockIdx.x, h = blockIdx.y;
  const int start = a.cu_seqlens[b], n_rows = a.cu_seqlens[b + 1] - start;
  if (n_rows <= 0 || a.token_req[start] < 0) {
    pdl_wait();
    return;
  }
  const int lane = threadIdx.x & 31, j = threadIdx.x % kLanes, pair = threadIdx.x / kLanes;
  const int c0 = blockIdx.z * kCols + kE * pair;
  const int D = a.D, V = a.V, rec = a.rec, at = delta_scalars_at(D);
  const int phase = a.state_phase[b];
  const float* old = a.state + (size_t)a.state_slots[b] * a.state_stride + ((size_t)phase * a.H + h) * D * V;
  float* fresh = a.state + (size_t)a.state_slots[b] * a.state_stride + ((size_t)(1 - phase) * a.H + h) * D * V;
  pdl_wait();    // ahead of it the metadata alone: the old state may be what the kernel before leaves behind
  float C[kE][R];
#pragma unroll
  for (int e = 0; e < kE; ++e)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int d = channel_of<kLanes, kVec4>(i, j);
      C[e][i] = (c0 + e < V && d < D) ? old[(size_t)(c0 + e) * D + d] : 0.f;
    }
  // which of a run's sums this lane ends up with, and where the sums with the keys of its column are
  const int my_col = (j / (kLanes / 2)) & 1, my_row = (j / kRowStep) & 3;
  const bool writer = ((j / kKindStep) & 1) != 0 && j % kKindStep == 0;      // one of the lanes with the sum with a query
  const int key_src = (lane & ~(kLanes - 1)) + my_col * (kLanes / 2);
  const int buf_floats = chunk * (rec + kCols);
  auto request = [&](int t0, int buf) {
    const int n = min(chunk, n_rows - t0), rec4 = rec / 4;
    float* st = stage + (size_t)buf * buf_floats;
    float* vl = st + (size_t)chunk * rec;
    const float* src = a.prep + ((size_t)h * a.tokens + start + t0) * rec;       // a head's records follow one another
    for (int i = threadIdx.x; i < n * rec4; i += kThreads) cp_async<16>(st + 4 * i, src + 4 * i);
    for (int i = threadIdx.x; i < n * kCols; i += kThreads) {
      const int tt = i / kCols, cc = blockIdx.z * kCols + (i - tt * kCols);
      if (cc < V) cp_async<4>(vl + i, a.qkv + (size_t)(start + t0 + tt) * a.ld_qkv + a.v_off + h * V + cc);
      else vl[i] = 0.f;
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  request(0, 0);
  int turn = 0;
  for (int t0 = 0; t0 < n_rows; t0 += chunk, turn ^= 1) {      // chunk: a multiple of four, so that runs do not straddle it
    const int n = min(chunk, n_rows - t0);
    if (t0 + chunk < n_rows) {
      request(t0 + chunk, turn ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const float* stage_now = stage + (size_t)turn * buf_floats;
    const float* vals = stage_now + (size_t)chunk * rec;
    int tt = 0;
#pragma unroll 2
    for (; tt + 3 < n; tt += 4) {
      const float* run = stage_now + (size_t)tt * rec;
      float k[4][R], v[8 * kE];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float q[R];
        load_channels<kLanes, R, kVec4>(k[u], run + (size_t)u * rec, D, j);
        load_channels<kLanes, R, kVec4>(q, run + (size_t)u * rec + D, D, j);
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          float pk[2] = {0.f, 0.f}, pq[2] = {0.f, 0.f};
#pragma unroll
          for (int i = 0; i < R; ++i) {
            pk[i & 1] += C[e][i] * k[u][i];
            pq[i & 1] += C[e][i] * q[i];
          }
          v[(e * 4 + u) * 2] = pk[0] + pk[1];
          v[(e * 4 + u) * 2 + 1] = pq[0] + pq[1];
        }
      }
      // the run's numbers that wait for no sum
      float4 s0[4], s1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        s0[u] = *reinterpret_cast<const float4*>(run + (size_t)u * rec + at);       // beta, P, g, ck0
        s1[u] = *reinterpret_cast<const float4*>(run + (size_t)u * rec + at + 4);   // ck1, ck2, cq0, cq1
      }
      const float* own = run + (size_t)my_row * rec + at;
      const float own_P = own[1], cq0 = own[6], cq1 = own[7], cq2 = own[8], cq3 = own[9];
      const float4 tail = *reinterpret_cast<const float4*>(run + (size_t)3 * rec + at + 8);   // cq2, cq3, R_31, R_30
      float want[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) want[u] = vals[(tt + u) * kCols + kE * pair + my_col];
      // halving: column, row, row, kind
#pragma unroll
      for (int half = 4 * kE, o = kLanes / 2; half > 0; half >>= 1, o >>= 1) {
        const bool up = (j & o) != 0;
#pragma unroll
        for (int i = 0; i < 4 * kE; ++i)
          if (i < half) {
            const float send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
      }
#pragma unroll
      for (int o = kKindStep / 2; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      float ak[4], d[4], dx[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) ak[u] = __shfl_sync(0xffffffffu, v[0], key_src + u * kRowStep);
      d[0] = s0[0].x * (want[0] - s0[0].y * ak[0]);
      d[1] = s0[1].x * (want[1] - s0[1].y * ak[1] - s0[1].w * d[0]);
      d[2] = s0[2].x * (want[2] - s0[2].y * ak[2] - s0[2].w * d[0] - s1[2].x * d[1]);
      d[3] = s0[3].x * (want[3] - s0[3].y * ak[3] - s0[3].w * d[0] - s1[3].x * d[1] - s1[3].y * d[2]);
      if (writer && c0 + my_col < V)
        a.out[(size_t)(start + t0 + tt + my_row) * a.ld_out + (size_t)h * V + c0 + my_col] =
            own_P * v[0] + (cq0 * d[0] + cq1 * d[1]) + (cq2 * d[2] + cq3 * d[3]);
      d[0] *= tail.w, d[1] *= tail.z, d[2] *= s0[3].z;
#pragma unroll
      for (int u = 0; u < 4; ++u) dx[u] = __shfl_xor_sync(0xffffffffu, d[u], kLanes / 2);    // the other column's
      const float keep = s0[3].y;
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        const bool mine = my_col == e;
        const float w0 = mine ? d[0] : dx[0], w1 = mine ? d[1] : dx[1], w2 = mine ? d[2] : dx[2], w3 = mine ? d[3] : dx[3];
#pragma unroll
        for (int i = 0; i < R; ++i) C[e][i] = keep * C[e][i] + ((k[0][i] * w0 + k[1][i] * w1) + (k[2][i] * w2 + k[3][i] * w3));
      }
    }
    for (; tt < n; ++tt) {
      const float* r = stage_now + (size_t)tt * rec;
      const float beta = r[at], g = r[at + 2];
      float k[R], q[R];
      load_channels<kLanes, R, kVec4>(k, r, D, j);
      load_channels<kLanes, R, kVec4>(q, r + D, D, j);
#pragma unroll
      for (int e = 0; e < kE; ++e) {
        float kv[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < R; ++i) {
          C[e][i] *= g;
          kv[i & 1] += C[e][i] * k[i];
        }
        const float dlt = beta * (vals[tt * kCols + kE * pair + e] - lanes_sum<kLanes>(kv[0] + kv[1]));
        float num[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < R; ++i) {
          C[e][i] += k[i] * dlt;
          num[i & 1] += C[e][i] * q[i];
        }
        const float o = lanes_sum<kLanes>(num[0] + num[1]);
        if (j == 0 && c0 + e < V) a.out[(size_t)(start + t0 + tt) * a.ld_out + (size_t)h * V + c0 + e] = o;
      }
    }
    __syncthreads();                           // everyone has read this buffer before the chunk after next is requested into it
  }
#pragma unroll
  for (int e = 0; e < kE; ++e)
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int d = channel_of<kLanes, kVec4>(i, j);
      if (c0 + e < V && d < D) fresh[(size_t)(c0 + e) * D + d] = C[e][i];
    }
}

// out[t, h, c] = o[t, h, c] * rsqrt(mean_c o[t, h, :]^2 + eps) * w[h * w_stride + c] * act(gate[t, h, c]) * scale, act the
// sigmoid (gate_act OI_ACT_NONE) or silu (OI_ACT_SILU):
// the per-head unit norm, the weight and the output gate of a recurrent mixer, one warp per (row, head).
template <typename TO>
__global__ void head_norm_gate_kernel(TO* __restrict__ out, long long ld_out, const float* __restrict__ o, long long ld_o,
                                      const float* __restrict__ gate, long long ld_gate, const void* __restrict__ w,
                                      int w_dtype, int w_stride, int tokens, int H, int V, float eps, float scale, int gate_act) {
  pdl_start();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= tokens * H) return;
  const int t = warp / H, h = warp - t * H;
  const float* row = o + (size_t)t * ld_o + (size_t)h * V;
  float ss = 0.f;
  for (int c = lane; c < V; c += 32) ss += row[c] * row[c];
  ss = warp_sum(ss);
  const float r = 1.f / sqrtf(ss / (float)V + eps);
  for (int c = lane; c < V; c += 32) {
    const float gz = gate[(size_t)t * ld_gate + (size_t)h * V + c];
    const float val = row[c] * r * load_as_f32(w, w_dtype, (size_t)h * w_stride + c) * gate_value(gz, gate_act) * scale;
    out[(size_t)t * ld_out + (size_t)h * V + c] = from_f32<TO>(val);
  }
}

// The same for ONE norm over a whole row of many numbers (H = 1: a norm over all heads together): one block a row.
template <typename TO>
__global__ void row_norm_gate_kernel(TO* __restrict__ out, long long ld_out, const float* __restrict__ o, long long ld_o,
                                     const float* __restrict__ gate, long long ld_gate, const void* __restrict__ w, int w_dtype,
                                     int V, float eps, float scale, int gate_act) {
  pdl_start();
  __shared__ float red[32];
  const int t = blockIdx.x;
  const float* row = o + (size_t)t * ld_o;
  float ss = 0.f;
  for (int c = threadIdx.x; c < V; c += blockDim.x) ss += row[c] * row[c];
  ss = block_sum(ss, red);
  const float r = 1.f / sqrtf(ss / (float)V + eps);
  for (int c = threadIdx.x; c < V; c += blockDim.x) {
    const float gz = gate[(size_t)t * ld_gate + c];
    out[(size_t)t * ld_out + c] = from_f32<TO>(row[c] * r * load_as_f32(w, w_dtype, c) * gate_value(gz, gate_act) * scale);
  }
}

}  // namespace

// floats of scratch the scan wants per row: oi_recurrent_scan's `prep` is [tokens, H, that]
OI_API int oi_recurrent_record(int mode, int D) {                        // a multiple of four floats: 16-byte copies
  if (mode == kGatedDelta) return run_row(D) + padded4(D);      // (a run of one row has its decay products behind it)
  return mode == kDeltaHeadDecay ? delta_scalars_at(D) + kDeltaScalars : (3 * D + 2 + 3) & ~3;
}

// mode 0: matrix memory (p0, p1: the two gate biases [H]); mode 1: gated delta rule (p0: dt [H * D], p1: A [H];
// decay: a [tokens, ld_decay]); mode 3: the delta rule with one decay per head (a at f_off of `gates`, p0: dt [H], p1: A [H]); mode 2: linear attention with a fixed decay per head (p0: lambda [H]; qkv is written: the
// values get their silu in place). State: [slots][2][H][D * V (+ D + 1 in mode 0)] floats. prep: scratch, see above.
OI_API int oi_recurrent_scan(int mode, const float* qkv, long long ld_qkv, int q_off, int k_off, int v_off, const float* gates,
                             long long ld_gates, int i_off, int f_off, const float* decay, long long ld_decay, const void* p0,
                             const void* p1, int p_dtype, float cap, float q_scale, float* prep, float* state,
                             long long state_stride, const int* cu_seqlens, const int* token_req, const int* state_slots,
                             const int* state_phase, float* out, long long ld_out, int tokens, int requests, int H, int G, int D,
                             int V, void* stream) {
  OI_REQUIRE(mode == kMatrixMemory || mode == kGatedDelta || mode == kLinearDecay || mode == kDeltaHeadDecay, "recurrent_scan: unknown mode %d", mode);
  OI_REQUIRE(requests >= 0 && tokens >= 0 && H > 0 && G > 0 && H % G == 0 && D > 0 && V > 0,
             "recurrent_scan: bad sizes H=%d G=%d D=%d V=%d", H, G, D, V);
  OI_REQUIRE(D <= 32 * kMaxRegs, "recurrent_scan: %d key channels per head, at most %d", D, 32 * kMaxRegs);
  OI_REQUIRE(mode != kGatedDelta || decay != nullptr, "recurrent_scan: the delta rule needs its decays");
  OI_REQUIRE(prep != nullptr, "recurrent_scan: the scratch for the rows' records is missing");
  const long long elems = (long long)D * V + (mode == kMatrixMemory ? D + 1 : 0);
  OI_REQUIRE(state != nullptr && state_stride >= 2 * H * elems, "recurrent_scan: the state needs two copies of %lld floats per head", elems);
  if (requests == 0 || tokens == 0) return OI_OK;
  ScanArgs a;
  a.qkv = qkv, a.ld_qkv = ld_qkv, a.q_off = q_off, a.k_off = k_off, a.v_off = v_off;
  a.gates = gates, a.ld_gates = ld_gates, a.i_off = i_off, a.f_off = f_off;
  a.decay = decay, a.ld_decay = ld_decay, a.p0 = p0, a.p1 = p1, a.p_dtype = p_dtype, a.cap = cap, a.q_scale = q_scale;
  a.prep = prep, a.rec = oi_recurrent_record(mode, D);
  a.state = state, a.state_stride = state_stride, a.cu_seqlens = cu_seqlens, a.token_req = token_req;
  a.state_slots = state_slots, a.state_phase = state_phase, a.out = out, a.ld_out = ld_out;
  a.tokens = tokens, a.H = H, a.G = G, a.D = D, a.V = V;
  cudaStream_t s = (cudaStream_t)stream;
  const int warps = tokens * H;
  if (mode == kMatrixMemory) oi_launch(recurrent_prepare_kernel<kMatrixMemory>, (warps + 3) / 4, 128, 0, s, a);
  else if (mode == kLinearDecay) oi_launch(recurrent_prepare_kernel<kLinearDecay>, (warps + 3) / 4, 128, 0, s, a);
  else if (mode == kDeltaHeadDecay) oi_launch(delta_head_prepare_kernel, (warps + 3) / 4, 128, 0, s, a);
  else oi_launch(D <= 128 ? delta_channel_prepare_kernel<4> : (D <= 256 ? delta_channel_prepare_kernel<8> : delta_channel_prepare_kernel<16>),
                 (warps + 3) / 4, 128, 0, s, a);
  OI_CHECK_LAUNCH();
  // Requests of several rows in plain stream order: launched early, the few long-lived blocks would be packed onto the SMs that
  // the kernel before frees first and share their issue slots (measured 2.1 against 0.9 ms for 2,048 rows). Single rows have no
  // such loop: launched early they find their place while the records are formed.
  const bool single = tokens == requests;
  if (mode == kDeltaHeadDecay) {
    const int rows = D <= 128 ? 16 : (D <= 256 ? 8 : 4);       // per buffer: two buffers of at most 19 KB
#define OI_DELTA_HEAD(LANES, REGS)                                                                                          \
  do {                                                                                                                      \
    constexpr int cols = 2 * kThreads / LANES;                                                                              \
    const dim3 grid(requests, H, (V + cols - 1) / cols);                                                                    \
    const size_t smem = 2 * (size_t)rows * (a.rec + cols) * sizeof(float);                                                  \
    if (!single) oi_fence_next_launch();                                                                                    \
    if (D % 4 == 0) oi_launch(delta_head_scan_kernel<LANES, REGS, true>, grid, kThreads, smem, s, a, rows);                 \
    else oi_launch(delta_head_scan_kernel<LANES, REGS, false>, grid, kThreads, smem, s, a, rows);                           \
  } while (0)
    // (one column a lane, twice the blocks, measured a tenth slower for 2,048 rows of 8 heads of 128 keys and values)
    if (D <= 64) OI_DELTA_HEAD(16, 4);
    else if (D <= 128) OI_DELTA_HEAD(32, 4);
    else if (D <= 256) OI_DELTA_HEAD(32, 8);
    else OI_DELTA_HEAD(32, 16);
#undef OI_DELTA_HEAD
    OI_CHECK_LAUNCH();
    return OI_OK;
  }
  // Lanes a column where either form takes the head: with eight an SM's schedulers issue least, with sixteen a run's chain is
  // shorter and there are twice the blocks, which counts while the blocks of eight lanes would be fewer than three for two SMs.
  // us with 8 / 16 lanes, 8 heads, requests of up to 1,500 rows (the records included): delta rule (128 values) 1 request 425 / 316,
  // 4 458 / 435, 6 (192 blocks of eight lanes) 625 / 572, 8 (256) 645 / 786, 16 1,095 / 1,255; matrix memory (256 values) 1 request
  // 453 / 377, 2 471 / 493, 3 (192) 650 / 640, 4 (256) 660 / 821, 16 1,927 / 2,351. The two add a row's products in another order, so
  // in batch-invariant mode it is eight whatever the step; the linear decay takes sixteen whatever the step (up to 2,000 rows:
  // 1 request 426 / 349, 4 458 / 468, 8 657 / 753).
  const bool few = !oi_option(OI_OPT_BATCH_INVARIANT) && (long long)requests * H * ((V + 31) / 32) < 222;
  if (mode == kGatedDelta) {
    const int rows = D <= 128 ? 16 : 4;                         // per buffer: two buffers of at most 30 KB
#define OI_DELTA_CHANNEL(LANES, REGS)                                                                                       \
  do {                                                                                                                      \
    constexpr int cols = 2 * kThreads / LANES;                                                                              \
    const dim3 grid(requests, H, (V + cols - 1) / cols);                                                                    \
    const size_t smem = 2 * ((size_t)(rows / 4) * (4 * run_row(D) + padded4(D)) + rows * cols) * sizeof(float);             \
    if (!single) oi_fence_next_launch();                                                                                    \
    auto kernel = D % 4 == 0 ? delta_channel_scan_kernel<LANES, REGS, true> : delta_channel_scan_kernel<LANES, REGS, false>; \
    if (smem > 48 * 1024) OI_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    oi_launch(kernel, grid, kThreads, smem, s, a, rows);                                                                    \
  } while (0)
    if (D <= 32) OI_DELTA_CHANNEL(8, 4);
    else if (D <= 64) OI_DELTA_CHANNEL(16, 4);
    else if (D <= 128 && few) OI_DELTA_CHANNEL(16, 8);
    else if (D <= 128) OI_DELTA_CHANNEL(8, 16);
    else if (D <= 256) OI_DELTA_CHANNEL(32, 8);
    else OI_DELTA_CHANNEL(32, 16);
#undef OI_DELTA_CHANNEL
    OI_CHECK_LAUNCH();
    return OI_OK;
  }
  // rows per buffer, a multiple of the four that are walked together: two buffers of at most 28 KB
  const int chunk = D <= 128 ? 16 : 4;
#define OI_SCAN_AS(MODE, LANES, REGS)                                                                                   \
  do {                                                                                                                  \
    constexpr int cols = 2 * kThreads / LANES;                                                                          \
    const dim3 grid(requests, H, (V + cols - 1) / cols);                                                                \
    const size_t smem = 2 * (size_t)chunk * (a.rec + cols) * sizeof(float);                                                 \
    if (!single) oi_fence_next_launch();                                                                                \
    auto kernel = D % 4 == 0 ? recurrent_scan_kernel<MODE, LANES, REGS, true> : recurrent_scan_kernel<MODE, LANES, REGS, false>; \
    if (smem > 48 * 1024) OI_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); \
    oi_launch(kernel, grid, kThreads, smem, s, a, chunk);                                                               \
  } while (0)
#define OI_SCAN(MODE, UP_TO_128)                 \
  do {                                           \
    if (D <= 32) OI_SCAN_AS(MODE, 8, 4);         \
    else if (D <= 64) OI_SCAN_AS(MODE, 16, 4);   \
    else if (D <= 128) UP_TO_128;                \
    else if (D <= 256) OI_SCAN_AS(MODE, 32, 8);  \
    else OI_SCAN_AS(MODE, 32, 16);               \
  } while (0)
  if (mode == kLinearDecay) OI_SCAN(kLinearDecay, OI_SCAN_AS(kLinearDecay, 16, 8));
  else if (few) OI_SCAN(kMatrixMemory, OI_SCAN_AS(kMatrixMemory, 16, 8));
  else OI_SCAN(kMatrixMemory, OI_SCAN_AS(kMatrixMemory, 8, 16));
#undef OI_SCAN
#undef OI_SCAN_AS
  OI_CHECK_LAUNCH();
  return OI_OK;
}

OI_API int oi_head_norm_gate(void* out, int out_dtype, long long ld_out, const float* o, long long ld_o, const float* gate,
                             long long ld_gate, const void* w, int w_dtype, int w_stride, int tokens, int H, int V, float eps,
                             float scale, int gate_act, void* stream) {
  OI_REQUIRE(tokens >= 0 && H > 0 && V > 0 && (gate_act == OI_ACT_NONE || gate_act == OI_ACT_SILU), "head_norm_gate: bad sizes or gate");
  if (tokens == 0) return OI_OK;
  const int warps = tokens * H, blocks = (warps + 7) / 8;
  cudaStream_t s = (cudaStream_t)stream;
  if (H == 1 && V >= 256 && (out_dtype == OI_F32 || out_dtype == OI_BF16)) {     // one long row: a block a row, not a warp
    const int threads = V >= 1024 ? 256 : 128;
    if (out_dtype == OI_F32)
      oi_launch(row_norm_gate_kernel<float>, tokens, threads, 0, s, (float*)out, ld_out, o, ld_o, gate, ld_gate, w, w_dtype, V, eps, scale, gate_act);
    else
      oi_launch(row_norm_gate_kernel<bf16>, tokens, threads, 0, s, (bf16*)out, ld_out, o, ld_o, gate, ld_gate, w, w_dtype, V, eps, scale, gate_act);
    OI_CHECK_LAUNCH();
    return OI_OK;
  }
  if (out_dtype == OI_F32)
    oi_launch(head_norm_gate_kernel<float>, blocks, 256, 0, s, (float*)out, ld_out, o, ld_o, gate, ld_gate, w, w_dtype, w_stride, tokens, H, V, eps, scale, gate_act);
  else if (out_dtype == OI_BF16)
    oi_launch(head_norm_gate_kernel<bf16>, blocks, 256, 0, s, (bf16*)out, ld_out, o, ld_o, gate, ld_gate, w, w_dtype, w_stride, tokens, H, V, eps, scale, gate_act);
  else
    OI_REQUIRE(false, "head_norm_gate: unknown dtype code %d", out_dtype);
  OI_CHECK_LAUNCH();
  return OI_OK;
}
