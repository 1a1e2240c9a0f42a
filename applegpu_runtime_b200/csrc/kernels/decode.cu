// Kernels of the static-shape decode step (one new token per sequence against a preallocated KV cache).
//
// The reference appends to its KV cache by concatenation and recomputes shapes every step
// (python/applegpu_runtime/models/gpt2.py:122-135: concat(dim=1) of the cached and the new keys / values, then the
// non-causal `attention` composition over the grown tensors). Here the cache is a fixed [B, heads, T_max, 64]
// buffer per layer, the current length lives in device memory, and one kernel per layer writes the new key / value
// row in place and attends over rows 0 .. len: the step has the same launch list at every length, so it can be
// captured once as a CUDA graph and replayed.
#include "common.cuh"
#include "mma_sync.cuh"
#include "sm100.cuh"

namespace ag { namespace k {

float* skinny_partials();            // workspace.cu: created with the device context (shared with the skinny matmul)

__device__ __forceinline__ unsigned long long globaltimer_ns_dec() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Geometry of a split-K linear work item of a decode step (see decode_linear_kernel below).
constexpr int kDlCols = 64;       // columns per CTA
constexpr int kDlRows = 128;      // K rows per CTA
constexpr int kDlThreads = 256;
constexpr int kDlMaxM = 16;

// One (sequence, head) of a decode step's attention, by a block of kDlThreads threads.
// s_qkv: this head's q | k | v of the new token as floats that hold storage-type values; kc / vc: the head's cache
// [t_max, 64]; out_row: 64 outputs; len = tokens already in the cache (the new token becomes row len).
// A thread has one key of each 256 for the scores, and for the weighted sum 16 bytes of the rows of one key in 256 / (threads
// that share a row); the first 256 keys' pieces of both are asked for before anything else (AttnDecodeRegs). What bounds it is the
// chain of L2 round trips of one block, so nothing is read twice and no load waits for a sum: 7.4 -> 3.8 us a launch at 8 x 12
// heads and 64 to 114 keys.
struct AttnDecodeSmem {
  float s_q[64];
  float s_o[kDlThreads / 32][64];
  float s_red[33];
};
template <typename T> struct AttnDecodeRegs {
  static constexpr int kPacks = 64 / Pack<T>::N;              // 16-byte pieces of a row
  static constexpr int kGroups = kDlThreads / kPacks;         // keys whose values are read at once
  static constexpr int kPre = 8;                              // rounds of them asked for ahead
  Pack<T> k[kPacks], v[kPre];
};
__device__ __forceinline__ int attn_decode_len(int len, int t_max) { return len < 0 ? 0 : len > t_max - 1 ? t_max - 1 : len; }   // a full cache overwrites its last row
template <typename T>
__device__ __forceinline__ void attn_decode_fetch(const T* kc, const T* vc, int len, AttnDecodeRegs<T>& r) {
  using R = AttnDecodeRegs<T>;
  const int tid = threadIdx.x, grp = tid / R::kPacks, c = tid % R::kPacks;
  if (tid < len) {
#pragma unroll
    for (int i = 0; i < R::kPacks; i++) r.k[i] = ld16(kc + (long long)tid * 64 + i * Pack<T>::N);
  }
#pragma unroll
  for (int i = 0; i < R::kPre; i++) if (grp + i * R::kGroups < len) r.v[i] = ld16(vc + (long long)(grp + i * R::kGroups) * 64 + c * Pack<T>::N);
}
template <typename T>
__device__ __forceinline__ void attn_decode_item(const float* s_qkv, T* kc, T* vc, T* out_row, int len, float scale, float* s_scores, AttnDecodeSmem& sm, AttnDecodeRegs<T>& pre) {
  using R = AttnDecodeRegs<T>;
  constexpr int N = Pack<T>::N;
  const int tid = threadIdx.x;
  // append the new key / value row in place; q pre-scaled. Nothing below reads the new row from global memory.
  if (tid < 64) { kc[(long long)len * 64 + tid] = Cvt<T>::from(s_qkv[64 + tid]); sm.s_q[tid] = s_qkv[tid] * scale; }
  else if (tid < 128) vc[(long long)len * 64 + (tid - 64)] = Cvt<T>::from(s_qkv[128 + (tid - 64)]);
  __syncthreads();
  float m_local = -INFINITY;
  for (int j = tid; j <= len; j += kDlThreads) {
    float acc = 0.f;
    if (j == len) {
      for (int c = 0; c < 64; c++) acc = fmaf(sm.s_q[c], s_qkv[64 + c], acc);
    } else {
      if (j != tid) {
#pragma unroll
        for (int i = 0; i < R::kPacks; i++) pre.k[i] = ld16(kc + (long long)j * 64 + i * N);
      }
#pragma unroll
      for (int i = 0; i < R::kPacks; i++)
#pragma unroll
        for (int e = 0; e < N; e++) acc = fmaf(sm.s_q[i * N + e], Cvt<T>::to(pre.k[i].v[e]), acc);
    }
    s_scores[j] = acc;
    m_local = fmaxf(m_local, acc);
  }
  const float m = block_max(m_local, sm.s_red);
  float l_local = 0.f;
  for (int j = tid; j <= len; j += kDlThreads) { const float p = __expf(s_scores[j] - m); s_scores[j] = p; l_local += p; }
  const float l = block_sum(l_local, sm.s_red);          // its barriers make the weights visible as well
  const int grp = tid / R::kPacks, c = tid % R::kPacks;
  float o[N];
#pragma unroll
  for (int e = 0; e < N; e++) o[e] = 0.f;
#pragma unroll
  for (int i = 0; i < R::kPre; i++) {
    const int j = grp + i * R::kGroups;
    if (j < len) {
      const float p = s_scores[j];
#pragma unroll
      for (int e = 0; e < N; e++) o[e] = fmaf(p, Cvt<T>::to(pre.v[i].v[e]), o[e]);
    }
  }
#pragma unroll 4
  for (int j = grp + R::kPre * R::kGroups; j < len; j += R::kGroups) {
    const Pack<T> v = ld16(vc + (long long)j * 64 + c * N);
    const float p = s_scores[j];
#pragma unroll
    for (int e = 0; e < N; e++) o[e] = fmaf(p, Cvt<T>::to(v.v[e]), o[e]);
  }
  if (grp == len % R::kGroups) {
    const float p = s_scores[len];
#pragma unroll
    for (int e = 0; e < N; e++) o[e] = fmaf(p, s_qkv[128 + c * N + e], o[e]);
  }
#pragma unroll
  for (int e = 0; e < N; e++) {
#pragma unroll
    for (int d = R::kPacks; d < 32; d *= 2) o[e] += __shfl_xor_sync(0xffffffffu, o[e], d);
  }
  if ((tid & 31) < R::kPacks) {
#pragma unroll
    for (int e = 0; e < N; e++) sm.s_o[tid >> 5][c * N + e] = o[e];
  }
  __syncthreads();
  if (tid < 64) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kDlThreads / 32; w++) t += sm.s_o[w][tid];
    out_row[tid] = Cvt<T>::from(t / l);
  }
}

// grid = B * heads. qkv: [B, 3 * d] rows (q | k | v of the new token); caches: [B, heads, t_max, 64]; out: [B, d] (heads
// merged). *len_ptr = tokens already in the cache; the new token becomes row *len_ptr.
// The length and the cached rows are read before the dependency wait: the length is older than the launch before this one (the
// step's embedding and projection lie between, and every kernel of a step waits for the one before it ahead of letting the next one
// start), and so are the rows below it.
template <typename T>
__global__ void __launch_bounds__(kDlThreads) attention_decode_kernel(const T* __restrict__ qkv, T* kcache, T* vcache, T* __restrict__ out, const int* len_ptr, int heads, int t_max,
                                                                      float scale) {
  extern __shared__ float s_scores[];          // [t_max]
  __shared__ AttnDecodeSmem sm;
  __shared__ float s_qkv[192];
  const int b = blockIdx.x / heads, h = blockIdx.x % heads;
  const int d = heads * 64;
  T* kc = kcache + ((long long)b * heads + h) * (long long)t_max * 64;
  T* vc = vcache + ((long long)b * heads + h) * (long long)t_max * 64;
  const int len = attn_decode_len(*len_ptr, t_max);
  AttnDecodeRegs<T> pre;
  attn_decode_fetch<T>(kc, vc, len, pre);
  pdl_wait();
  pdl_trigger();
  const T* row = qkv + (long long)b * 3 * d;
  if (threadIdx.x < 192) s_qkv[threadIdx.x] = Cvt<T>::to(row[(threadIdx.x >> 6) * d + h * 64 + (threadIdx.x & 63)]);
  __syncthreads();
  attn_decode_item<T>(s_qkv, kc, vc, out + (long long)b * d + h * 64, len, scale, s_scores, sm, pre);
}

Status attention_decode(cudaStream_t s, DType dt, const void* qkv, void* kcache, void* vcache, void* out, const int* len_ptr, int batch, int heads, int t_max, float scale) {
  if (batch <= 0 || heads <= 0) return Status::OK();
  if (!qkv) return Status::invalid("attention_decode: no q / k / v");
  if (t_max <= 0 || t_max > 8192) return Status::invalid("attention_decode: cache length must be in 1..8192");
  if (!aligned16(kcache) || !aligned16(vcache)) return Status::compute("attention_decode needs 16-byte aligned caches");
  const size_t smem = (size_t)t_max * sizeof(float);
  cudaError_t le = cudaSuccess;
  AG_DISPATCH_FLOAT(dt, T, (le = launch_pdl(attention_decode_kernel<T>, dim3((unsigned)(batch * heads)), dim3(kDlThreads), smem, s, (const T*)qkv, (T*)kcache,
                                             (T*)vcache, (T*)out, len_ptr, heads, t_max, scale)));
  if (le != cudaSuccess) return cuda_status(le, "attention_decode");
  return Status::OK();
}

// ── linear layer of a decode step ───────────────────────────────────────────
// y[M, N] = act(layer_norm?(x)[M, K] @ W[K, N] + bias) + residual with M <= 16 and W as the reference stores its
// Conv1D weights ([in, out], rows along N). The product reads W once, and what a launch takes is the chain of round trips behind
// its inputs, so:
//   * a CTA has 64 columns and a share of K in slabs of 128 rows; the (at most eight) shares of a column slab are a cluster, whose
//     sums meet over distributed shared memory in K order: no partials in global memory, no fence, counter and reload;
//   * W is a model weight, never written by a kernel of the step, so its loads are issued BEFORE the programmatic
//     dependency wait: they overlap the previous kernel's tail, and x (which that kernel produces) is read after it;
//   * layer_norm of x runs in the prologue: every CTA takes the row statistics over the whole rows itself
//     (kernel_templates.rs:1097-1109: mean, population variance, 1/sqrt(var + eps)) and normalises its K share on the
//     way into shared memory, which removes the separate layer_norm launches of the step;
//   * 16-bit weights are multiplied by mma.m16n8k16 from registers (dl_products16). Stored inputs have the weight's type and enter as they
//     are; a normalised input is float32 and enters as the sum of three 16-bit numbers (DlSplit). float32 weights keep CUDA-core
//     multiply-adds.
// Every thread runs this code once per launch, so a launch takes about as long as its instructions: options are template parameters and
// nothing is unrolled beyond what the shape needs. GPT-2 small, 8 rows, bf16, a launch's share of a replayed step: 7.8 us with
// multiply-adds, partials in the L2 and a last CTA that adds them; 7.9 us with cluster sums and MMAs but x through shared memory and one
// kernel for all options (38 to 68 KB of code); now 3.5 (no layer_norm), 3.6 (K = 3072) and 4.8 us (layer_norm), 12 to 20 KB. Four shares
// in place of eight: 25 against 23 ms a generation, measured with the second form.

struct DecodeLinearParams {
  const void* x; const void* w; void* y;
  const void* bias; const void* residual; const void* ln_gamma; const void* ln_beta;
  float ln_eps; int act;
  int m, n, k;
  long long x_row, w_row, y_row;
  // the persistent engine only:
  float* partial;            // [shares][16][n]
  // x not materialised: it is act(sum over xp_shares of xp[share][m][.] + xp_bias) rounded to the storage type, i.e. the
  // unfinished result of the previous linear of the step (its row length is this linear's k)
  const float* xp = nullptr; int xp_shares = 0; const void* xp_bias = nullptr; int xp_act = 0;
};

constexpr int kDlShares = 8;      // shares of K at most: a cluster of portable size
__host__ __device__ __forceinline__ int dl_per(int slabs) { return (slabs + kDlShares - 1) / kDlShares; }       // slabs of one share
__host__ __device__ __forceinline__ int dl_shares(int k) { const int slabs = (k + kDlRows - 1) / kDlRows, per = dl_per(slabs); return (slabs + per - 1) / per; }

constexpr int kDlXPad = 16, kDlSumPitch = kDlCols + 4;       // floats; keep the 16-byte accesses of eight lanes on different banks
// Shared memory of one linear work item of the persistent engine (a 64-column x 128-row slab of W against all rows of x).
struct DlStats { float mean[kDlMaxM], rstd[kDlMaxM]; };
struct DlSmem {
  alignas(16) float sX[kDlMaxM][kDlRows + kDlXPad];       // float32 weights: this item's slab of x (normalised if asked)
  alignas(16) float sSum[kDlThreads / 32][kDlMaxM][kDlSumPitch];
  DlStats st;
};

// A slab's weights: a warp owns 16 consecutive K rows. 16-bit: a lane has eight consecutive columns of four of them; float32: four
// columns of eight.
template <typename T> constexpr int kDlWv = sizeof(T) == 4 ? 8 : 4;
template <typename T>
__device__ __forceinline__ void dl_load_weights(const DecodeLinearParams& p, int n0, int k0, uint4 (&wv)[kDlWv<T>]) {
  const T* W = reinterpret_cast<const T*>(p.w);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (sizeof(T) == 4) {
    const int col = n0 + (lane & 15) * 4;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int kk = k0 + warp * 16 + i * 2 + (lane >> 4);
      wv[i] = kk < p.k && col < p.n ? __ldcs(reinterpret_cast<const uint4*>(W + (long long)kk * p.w_row + col)) : make_uint4(0u, 0u, 0u, 0u);
    }
  } else {
    const bool wide = ((reinterpret_cast<uintptr_t>(W) | (uintptr_t)(p.w_row * 2)) & 15u) == 0;
    const int col = n0 + (lane >> 2) * 8;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int kk = k0 + warp * 16 + (lane & 3) * 4 + i;
      const T* at = W + (long long)kk * p.w_row + col;
      wv[i] = make_uint4(0u, 0u, 0u, 0u);
      if (kk >= p.k) continue;
      if (wide && col + 8 <= p.n) wv[i] = __ldcs(reinterpret_cast<const uint4*>(at));
      else {                                             // rows on 8 bytes, or half a piece at the end of one
        if (col < p.n) { const uint2 u = __ldcs(reinterpret_cast<const uint2*>(at)); wv[i].x = u.x; wv[i].y = u.y; }
        if (col + 4 < p.n) { const uint2 u = __ldcs(reinterpret_cast<const uint2*>(at + 4)); wv[i].z = u.x; wv[i].w = u.y; }
      }
    }
  }
}

// Row statistics of layer_norm over the whole rows of x: a warp per row, the row in registers after one round of
// 16-byte loads (kernel_templates.rs:1097-1109: mean, population variance, 1/sqrt(var + eps)). Ends with a block barrier.
// IT: 32 x 16-byte rounds of a row at most; what lies behind them would be left out.
template <typename T, int IT = 8>
__device__ __forceinline__ void dl_ln_stats(const DecodeLinearParams& p, DlStats& sm) {
  constexpr int N16 = Pack<T>::N;
  const T* X = reinterpret_cast<const T*>(p.x);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int m = warp; m < p.m; m += kDlThreads / 32) {
    const T* xr = X + (long long)m * p.x_row;
    const int packs = p.k / N16;
    Pack<T> q[IT];
    float sum = 0.f;
#pragma unroll
    for (int it = 0; it < IT; it++) if (lane + it * 32 < packs) q[it] = ld16(xr + (lane + it * 32) * N16);
#pragma unroll
    for (int it = 0; it < IT; it++) {
      if (lane + it * 32 < packs) {
#pragma unroll
        for (int e = 0; e < N16; e++) sum += Cvt<T>::to(q[it].v[e]);
      }
    }
    const float mean = warp_sum(sum) / (float)p.k;
    float sq = 0.f;
#pragma unroll
    for (int it = 0; it < IT; it++) {
      if (lane + it * 32 < packs) {
#pragma unroll
        for (int e = 0; e < N16; e++) { const float dlt = Cvt<T>::to(q[it].v[e]) - mean; sq += dlt * dlt; }
      }
    }
    const float var = warp_sum(sq) / (float)p.k;
    if (lane == 0) { sm.mean[m] = mean; sm.rstd[m] = 1.0f / sqrtf(var + p.ln_eps); }
  }
  __syncthreads();
}

// 128 columns of x from k0 on go into shared memory as floats, layer_norm applied on the way if asked. A thread has eight columns of
// one row: dl_ask_norm and dl_ask_x ask for them (the former before the dependency wait: gamma and beta are model weights), dl_put_x
// writes them once the statistics are there. K is a multiple of eight.
constexpr int kDlPer = kDlRows / 16;
template <typename T> struct DlX { Pack<T> x[kDlPer / Pack<T>::N], g[kDlPer / Pack<T>::N], b[kDlPer / Pack<T>::N]; };
__device__ __forceinline__ int dl_x_col(int k0) { return k0 + (threadIdx.x & 15) * kDlPer; }
template <typename T>
__device__ __forceinline__ void dl_ask_norm(const DecodeLinearParams& p, int k0, DlX<T>& r) {
  const int kk = dl_x_col(k0);
  if (!p.ln_gamma || kk >= p.k) return;
  const T* G = reinterpret_cast<const T*>(p.ln_gamma) + kk;
  const T* B = reinterpret_cast<const T*>(p.ln_beta) + kk;
  constexpr int N = Pack<T>::N;
  if (((reinterpret_cast<uintptr_t>(G) | reinterpret_cast<uintptr_t>(B)) & 15u) == 0) {
#pragma unroll
    for (int i = 0; i < kDlPer / N; i++) { r.g[i] = ld16(G + i * N); r.b[i] = ld16(B + i * N); }
  } else {
#pragma unroll
    for (int i = 0; i < kDlPer / N; i++)
#pragma unroll
      for (int e = 0; e < N; e++) { r.g[i].v[e] = G[i * N + e]; r.b[i].v[e] = B[i * N + e]; }
  }
}
template <typename T>
__device__ __forceinline__ void dl_ask_x(const DecodeLinearParams& p, int k0, DlX<T>& r) {
  const int m = threadIdx.x >> 4, kk = dl_x_col(k0);
  if (m >= p.m || kk >= p.k) return;
  const T* src = reinterpret_cast<const T*>(p.x) + (long long)m * p.x_row + kk;
#pragma unroll
  for (int i = 0; i < kDlPer / Pack<T>::N; i++) r.x[i] = ld16(src + i * Pack<T>::N);
}
template <typename T, int ROWS = kDlMaxM, bool LN = true>
__device__ __forceinline__ void dl_put_x(const DecodeLinearParams& p, const DlStats& st, float* sX, int pitch, int k0, const DlX<T>& r) {
  const int m = threadIdx.x >> 4, kk = dl_x_col(k0);
  constexpr int N = Pack<T>::N;
  float v[kDlPer];
#pragma unroll
  for (int e = 0; e < kDlPer; e++) v[e] = 0.f;
  if (m < p.m && kk < p.k) {
#pragma unroll
    for (int e = 0; e < kDlPer; e++) v[e] = Cvt<T>::to(r.x[e / N].v[e % N]);
    if (LN && p.ln_gamma) {
      const float mean = st.mean[m], rstd = st.rstd[m];
#pragma unroll
      for (int e = 0; e < kDlPer; e++) v[e] = Cvt<T>::to(r.g[e / N].v[e % N]) * (v[e] - mean) * rstd + Cvt<T>::to(r.b[e / N].v[e % N]);
    }
  }
  if (m >= ROWS) return;
#pragma unroll
  for (int e = 0; e < kDlPer; e += 4) *reinterpret_cast<float4*>(sX + m * pitch + (threadIdx.x & 15) * kDlPer + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
}
// The persistent engine's x that is not materialised: the previous linear's partials, added in K order, + bias, activation, rounded as
// they would have been stored.
template <typename T>
__device__ __forceinline__ void dl_put_partials(const DecodeLinearParams& p, float* sX, int pitch, int k0) {
  const int m = threadIdx.x >> 4, kk = dl_x_col(k0);
  float v[kDlPer];
#pragma unroll
  for (int e = 0; e < kDlPer; e++) v[e] = 0.f;
  if (m < p.m && kk < p.k) {
    float4 q[kDlShares][2];                              // all loads are in flight before the first addition
#pragma unroll
    for (int ks = 0; ks < kDlShares; ks++) {
      if (ks < p.xp_shares) {
        const float4* src = reinterpret_cast<const float4*>(p.xp + ((long long)ks * kDlMaxM + m) * p.k + kk);
        q[ks][0] = __ldcg(src); q[ks][1] = __ldcg(src + 1);
      }
    }
#pragma unroll
    for (int ks = 0; ks < kDlShares; ks++) {
      if (ks < p.xp_shares) {
        v[0] += q[ks][0].x; v[1] += q[ks][0].y; v[2] += q[ks][0].z; v[3] += q[ks][0].w;
        v[4] += q[ks][1].x; v[5] += q[ks][1].y; v[6] += q[ks][1].z; v[7] += q[ks][1].w;
      }
    }
#pragma unroll
    for (int e = 0; e < kDlPer; e++) {
      if (p.xp_bias) v[e] += Cvt<T>::to(reinterpret_cast<const T*>(p.xp_bias)[kk + e]);
      v[e] = Cvt<T>::to(Cvt<T>::from(apply_act(v[e], (Act)p.xp_act)));
    }
  }
#pragma unroll
  for (int e = 0; e < kDlPer; e += 4) *reinterpret_cast<float4*>(sX + m * pitch + (threadIdx.x & 15) * kDlPer + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
}

// float32 weights: this warp's 16 rows of a slab against the staged x, added to acc (two columns' halves: see dl_store_f32).
template <int ROWS>
__device__ __forceinline__ void dl_products_f32(const float* sX, int pitch, const uint4 (&wv)[8], float (&acc)[ROWS][4]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float* at = sX + warp * 16 + i * 2 + (lane >> 4);
    const float* pr = reinterpret_cast<const float*>(&wv[i]);
#pragma unroll
    for (int m = 0; m < ROWS; m++) {
      const float a = at[m * pitch];                         // two addresses per warp (one per half): broadcasts
#pragma unroll
      for (int e = 0; e < 4; e++) acc[m][e] = fmaf(a, pr[e], acc[m][e]);
    }
  }
}
// the two half-warps hold different rows of the same columns
template <int ROWS>
__device__ __forceinline__ void dl_store_f32(float (&acc)[ROWS][4], float (*sSum)[ROWS][kDlSumPitch]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int m = 0; m < ROWS; m++) {
#pragma unroll
    for (int e = 0; e < 4; e++) acc[m][e] += __shfl_xor_sync(0xffffffffu, acc[m][e], 16);
    if (lane < 16) *reinterpret_cast<float4*>(&sSum[warp][m][lane * 4]) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
  }
}

// A normalised value r as three 16-bit numbers, r = pre (h0 + h1 / step + h2 / step^2).
// bfloat16 has float32's exponents: its pieces are eight bits each, cut off and so of the value's sign, and hold the 24 as they are. The
// NaN that arithmetic leaves has its payload in the upper half.
// float16: |r| <= 2^22 (sqrt(2048) times the largest gamma, plus the largest beta), so r / 2^7 <= 2^15 and, a remainder being at most
// 2^-11 of what it remains of, every piece stays in range. The pieces hold 2^-35 of r, or 2^-43 where that is more: float32's 2^-24 from
// |r| = 2^-18 on.
template <typename T> struct DlSplit { static constexpr float pre = 1.f, step = 1.f; };
template <> struct DlSplit<__half> { static constexpr float pre = 128.f, step = 4096.f; };
__device__ __forceinline__ void dl_split(float (&r)[4], uint32_t (&b)[3][2], __half) {
#pragma unroll
  for (int piece = 0; piece < 3; piece++)
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const __half2 h = __floats2half2_rn(r[2 * i], r[2 * i + 1]);
      const float2 f = __half22float2(h);
      b[piece][i] = *reinterpret_cast<const uint32_t*>(&h);
      r[2 * i] = (r[2 * i] - f.x) * DlSplit<__half>::step; r[2 * i + 1] = (r[2 * i + 1] - f.y) * DlSplit<__half>::step;
    }
}
__device__ __forceinline__ void dl_split(float (&r)[4], uint32_t (&b)[3][2], __nv_bfloat16) {
#pragma unroll
  for (int piece = 0; piece < 3; piece++) {
    b[piece][0] = __byte_perm(__float_as_uint(r[0]), __float_as_uint(r[1]), 0x7632); b[piece][1] = __byte_perm(__float_as_uint(r[2]), __float_as_uint(r[3]), 0x7632);
#pragma unroll
    for (int e = 0; e < 4; e++) r[e] -= __uint_as_float(__float_as_uint(r[e]) & 0xffff0000u);
  }
}
template <typename T> __device__ __forceinline__ uint32_t dl_pair(T lo, T hi) {
  return (uint32_t)*reinterpret_cast<const uint16_t*>(&lo) | ((uint32_t)*reinterpret_cast<const uint16_t*>(&hi) << 16);
}
template <typename T> __device__ __forceinline__ float dl_elem(uint2 v, int e) {
  const uint32_t w = e < 2 ? v.x : v.y;
  const uint16_t h = (uint16_t)(e & 1 ? w >> 16 : w & 0xffffu);
  return Cvt<T>::to(*reinterpret_cast<const T*>(&h));
}

// 16-bit weights: a lane (g, q) has rows 4q .. 4q + 3 of the warp's 16 and columns 8g .. 8g + 7. The order of K in a product and of the
// columns is free as long as both operands agree, so mma.m16n8k16 takes the weights as they lie: product j has columns 8g + j and
// 8g + j + 4 in its rows, eight rows of x in its columns and the lane's four rows as its K, and the x operand is four neighbouring
// elements of row g, straight from memory.
__device__ __forceinline__ int dl_k_of(int k0) { return k0 + (threadIdx.x >> 5) * 16 + (threadIdx.x & 3) * 4; }
template <typename T>
__device__ __forceinline__ uint2 dl_ask4(const void* base, long long at) { return *reinterpret_cast<const uint2*>(reinterpret_cast<const T*>(base) + at); }
template <typename T, int NT>
__device__ __forceinline__ void dl_ask_x16(const DecodeLinearParams& p, int k0, uint2 (&x)[NT]) {
  const int kk = dl_k_of(k0), g = (threadIdx.x & 31) >> 2;
#pragma unroll
  for (int t = 0; t < NT; t++) x[t] = kk < p.k && g + 8 * t < p.m ? dl_ask4<T>(p.x, (long long)(g + 8 * t) * p.x_row + kk) : make_uint2(0u, 0u);
}
template <typename T>
__device__ __forceinline__ void dl_ask_norm16(const DecodeLinearParams& p, int k0, uint2& gam, uint2& bet) {
  const int kk = dl_k_of(k0);
  gam = make_uint2(0u, 0u); bet = gam;
  if (kk >= p.k) return;
  if (((reinterpret_cast<uintptr_t>(p.ln_gamma) | reinterpret_cast<uintptr_t>(p.ln_beta)) & 7u) == 0) { gam = dl_ask4<T>(p.ln_gamma, kk); bet = dl_ask4<T>(p.ln_beta, kk); return; }
  const T* G = reinterpret_cast<const T*>(p.ln_gamma) + kk;
  const T* B = reinterpret_cast<const T*>(p.ln_beta) + kk;
  gam.x = dl_pair(G[0], G[1]); gam.y = dl_pair(G[2], G[3]); bet.x = dl_pair(B[0], B[1]); bet.y = dl_pair(B[2], B[3]);
}
// LN: acc is in units of pre. An infinity or NaN is the first pieces' alone: what it leaves for the others, or an infinite weight times
// them, has no meaning.
template <typename T, int NT, bool LN>
__device__ __forceinline__ void dl_products16(const uint4 (&wv)[4], const uint2 (&x)[NT], uint2 gam, uint2 bet, const DlStats& st, float (&acc)[NT][4][4]) {
  const int g = (threadIdx.x & 31) >> 2;
  uint32_t a[4][4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    auto word = [&](int i, int c) { return c < 2 ? wv[i].x : c < 4 ? wv[i].y : c < 6 ? wv[i].z : wv[i].w; };
    const uint32_t sel = j & 1 ? 0x7632u : 0x5410u;
    a[j][0] = __byte_perm(word(0, j), word(1, j), sel); a[j][1] = __byte_perm(word(0, j + 4), word(1, j + 4), sel);
    a[j][2] = __byte_perm(word(2, j), word(3, j), sel); a[j][3] = __byte_perm(word(2, j + 4), word(3, j + 4), sel);
  }
#pragma unroll
  for (int t = 0; t < NT; t++) {
    if constexpr (!LN) {
#pragma unroll
      for (int j = 0; j < 4; j++) mma_16816<T>(acc[t][j], a[j][0], a[j][1], a[j][2], a[j][3], x[t].x, x[t].y);
    } else {
      const float mean = st.mean[g + 8 * t], rstd = st.rstd[g + 8 * t];
      float r[4];
#pragma unroll
      for (int e = 0; e < 4; e++) r[e] = (dl_elem<T>(gam, e) * (dl_elem<T>(x[t], e) - mean) * rstd + dl_elem<T>(bet, e)) * (1.f / DlSplit<T>::pre);
      uint32_t b[3][2];
      dl_split(r, b, T());
      float c[4][4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        c[j][0] = 0.f; c[j][1] = 0.f; c[j][2] = 0.f; c[j][3] = 0.f;
        mma_16816<T>(c[j], a[j][0], a[j][1], a[j][2], a[j][3], b[2][0], b[2][1]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) mma_16816<T>(acc[t][j], a[j][0], a[j][1], a[j][2], a[j][3], b[0][0], b[0][1]);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if constexpr (DlSplit<T>::step != 1.f) {
#pragma unroll
          for (int e = 0; e < 4; e++) c[j][e] *= 1.f / DlSplit<T>::step;
        }
        mma_16816<T>(c[j], a[j][0], a[j][1], a[j][2], a[j][3], b[1][0], b[1][1]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) if (isfinite(acc[t][j][e])) acc[t][j][e] = fmaf(c[j][e], 1.f / DlSplit<T>::step, acc[t][j][e]);
    }
  }
}
template <typename T, int NT>
__device__ __forceinline__ void dl_unit(float (&acc)[NT][4][4]) {
  if constexpr (DlSplit<T>::pre != 1.f) {
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[t][j][e] *= DlSplit<T>::pre;
  }
}
template <int NT>
__device__ __forceinline__ void dl_store16(const float (&acc)[NT][4][4], float (*sSum)[kDlSumPitch]) {     // this warp's [NT * 8][64]
  const int g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int h = 0; h < 2; h++) {                          // rows 2q and 2q + 1 of x; columns 8g + 0 .. 3, then 4 .. 7
      float* at = &sSum[t * 8 + q * 2 + h][g * 8];
      *reinterpret_cast<float4*>(at) = make_float4(acc[t][0][h], acc[t][1][h], acc[t][2][h], acc[t][3][h]);
      *reinterpret_cast<float4*>(at + 4) = make_float4(acc[t][0][h + 2], acc[t][1][h + 2], acc[t][2][h + 2], acc[t][3][h + 2]);
    }
}
template <int NT>
__device__ __forceinline__ void dl_zero(float (&acc)[NT][4][4]) {
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[t][j][e] = 0.f;
}

// The persistent engine's item: one share's partial product into p.partial[share][m][n0 ..]. Its sums are those of decode_linear_kernel,
// in the same order.
template <typename T>
__device__ __forceinline__ void dl_partial(const DecodeLinearParams& p, DlSmem& sm, int n0, int share, int per, uint4 (&wv)[kDlWv<T>]) {
  if constexpr (sizeof(T) == 4) {
    float acc[kDlMaxM][4];
#pragma unroll
    for (int m = 0; m < kDlMaxM; m++) { acc[m][0] = 0.f; acc[m][1] = 0.f; acc[m][2] = 0.f; acc[m][3] = 0.f; }
    for (int i = 0; i < per; i++) {
      const int k0 = (share * per + i) * kDlRows;
      if (i) { __syncthreads(); dl_load_weights<T>(p, n0, k0, wv); }
      if (p.xp) dl_put_partials<T>(p, &sm.sX[0][0], kDlRows + kDlXPad, k0);
      else {
        DlX<T> x;
        dl_ask_norm<T>(p, k0, x);
        dl_ask_x<T>(p, k0, x);
        dl_put_x<T>(p, sm.st, &sm.sX[0][0], kDlRows + kDlXPad, k0, x);
      }
      __syncthreads();
      dl_products_f32(&sm.sX[0][0], kDlRows + kDlXPad, wv, acc);
    }
    dl_store_f32(acc, sm.sSum);
  } else {
    float acc[2][4][4];
    dl_zero<2>(acc);
    for (int i = 0; i < per; i++) {
      const int k0 = (share * per + i) * kDlRows;
      if (i) dl_load_weights<T>(p, n0, k0, wv);
      uint2 x[2], gam = make_uint2(0u, 0u), bet = gam;
      if (p.xp) {                                          // values of type T again: dl_put_partials has rounded them
        __syncthreads();
        dl_put_partials<T>(p, &sm.sX[0][0], kDlRows + kDlXPad, k0);
        __syncthreads();
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int t = 0; t < 2; t++) {
          const float4 f = *reinterpret_cast<const float4*>(&sm.sX[(lane >> 2) + 8 * t][(threadIdx.x >> 5) * 16 + (lane & 3) * 4]);
          x[t] = make_uint2(dl_pair(Cvt<T>::from(f.x), Cvt<T>::from(f.y)), dl_pair(Cvt<T>::from(f.z), Cvt<T>::from(f.w)));
        }
      } else dl_ask_x16<T, 2>(p, k0, x);
      if (p.ln_gamma) { dl_ask_norm16<T>(p, k0, gam, bet); dl_products16<T, 2, true>(wv, x, gam, bet, sm.st, acc); }
      else dl_products16<T, 2, false>(wv, x, gam, bet, sm.st, acc);
    }
    if (p.ln_gamma) dl_unit<T, 2>(acc);
    dl_store16<2>(acc, sm.sSum[threadIdx.x >> 5]);
  }
  __syncthreads();
  float* my_partial = p.partial + ((long long)share * kDlMaxM) * p.n;
  for (int i = threadIdx.x; i < kDlMaxM * kDlCols; i += kDlThreads) {
    const int m = i / kDlCols, c = i % kDlCols;
    float v = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < kDlThreads / 32; w8++) v += sm.sSum[w8][m][c];      // warp order = K order
    if (m < p.m && n0 + c < p.n) my_partial[(long long)m * p.n + n0 + c] = v;
  }
}

// One finished element: the shares' partials added in K order (deterministic), bias, activation, residual.
template <typename T>
__device__ __forceinline__ float dl_finish_element(const DecodeLinearParams& p, int shares, int m, int col) {
  float v = 0.f;
  for (int ks = 0; ks < shares; ks++) v += __ldcg(p.partial + ((long long)ks * kDlMaxM + m) * p.n + col);
  if (p.bias) v += Cvt<T>::to(reinterpret_cast<const T*>(p.bias)[col]);
  v = apply_act(v, (Act)p.act);
  if (p.residual) v += Cvt<T>::to(reinterpret_cast<const T*>(p.residual)[(long long)m * p.y_row + col]);
  return v;
}

// The CTA's sums for its share (sSum, eight warps of them) to the results. Row m is finished by share m % shares: every CTA adds its warps'
// sums in K order and stores them in that CTA's sFin, and after one cluster barrier the finisher adds the shares in K order. The barrier
// that says the peers' shared memory exists was arrived at when the kernel started.
constexpr int kDlFinRows = kDlMaxM + kDlShares;            // shares x rows a share finishes, at most
template <typename T, int ROWS>
__device__ __forceinline__ void dl_finish(const DecodeLinearParams& p, int n0, int rank, int ranks, const float* sSum, float* sFin) {
  const int c = threadIdx.x & (kDlCols - 1), m0 = threadIdx.x / kDlCols;
  constexpr int STEP = kDlThreads / kDlCols;
  const int mine = (p.m - rank + ranks - 1) / ranks;       // rows this CTA finishes: rank, rank + ranks, ..
  const bool live = n0 + c < p.n;
  float bias = 0.f, res = 0.f;
  if (live && p.bias) bias = Cvt<T>::to(reinterpret_cast<const T*>(p.bias)[n0 + c]);
  if (live && p.residual && m0 < mine) res = Cvt<T>::to(reinterpret_cast<const T*>(p.residual)[(long long)(rank + m0 * ranks) * p.y_row + n0 + c]);
  if (ranks > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int per = (p.m + ranks - 1) / ranks;
#pragma unroll
  for (int j = 0; j < ROWS / STEP; j++) {
    const int m = m0 + j * STEP;
    if (m >= p.m) break;
    float v = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < kDlThreads / 32; w8++) v += sSum[(w8 * ROWS + m) * kDlSumPitch + c];      // warp order = K order
    float* at = sFin + (rank * per + m / ranks) * kDlCols + c;
    if (ranks > 1) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(sm100::mapa_u32(sm100::smem_u32(at), (uint32_t)(m % ranks))), "f"(v) : "memory");
    else *at = v;
  }
  if (ranks > 1) sm100::cluster_sync_all(); else __syncthreads();
  T* Y = reinterpret_cast<T*>(p.y);
  for (int i = m0; i < mine && live; i += STEP) {
    const int m = rank + i * ranks;
    float v = 0.f;
    for (int r = 0; r < ranks; r++) v += sFin[(r * per + i) * kDlCols + c];
    if (i != m0 && p.residual) res = Cvt<T>::to(reinterpret_cast<const T*>(p.residual)[(long long)m * p.y_row + n0 + c]);
    v = apply_act(v + bias, (Act)p.act);
    Y[(long long)m * p.y_row + n0 + c] = Cvt<T>::from(p.residual ? v + res : v);
  }
}

// grid = (column slabs, shares of K), a cluster per column slab; `per` slabs of 128 K rows in a share, PRE of them asked for ahead of the
// dependency wait (they are not produced by the step). NT groups of eight rows of x.
// LN: 0 or the rounds of layer_norm's statistics (IT above). Rows of up to 1024 columns are held to the registers of three CTAs an SM, so that the
// next launch's weights are under way beside this one: with 88 registers, two CTAs, 50 tokens of 8 sequences of GPT-2 small in bf16 take
// 16.7 ms in place of 14.7, and of 16 sequences 23.0 in place of 21.0.
template <typename T, int NT, int PRE, int LN>
__global__ void __launch_bounds__(kDlThreads, LN == 4 ? 3 : 0) decode_linear_kernel(const __grid_constant__ DecodeLinearParams p, int per) {
  __shared__ __align__(16) float sSum[kDlThreads / 32][NT * 8][kDlSumPitch];
  __shared__ float sFin[kDlFinRows * kDlCols];
  __shared__ DlStats st;
  const int ranks = gridDim.y, rank = ranks > 1 ? (int)sm100::cluster_ctarank() : 0;
  if (ranks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const int n0 = blockIdx.x * kDlCols, k0 = rank * per * kDlRows;
  uint4 wv[PRE][4];
  uint2 x[PRE][NT], gam[PRE], bet[PRE];
#pragma unroll
  for (int s = 0; s < PRE; s++) dl_load_weights<T>(p, n0, s < per ? k0 + s * kDlRows : p.k, wv[s]);
  if constexpr (LN) {
#pragma unroll
    for (int s = 0; s < PRE; s++) dl_ask_norm16<T>(p, s < per ? k0 + s * kDlRows : p.k, gam[s], bet[s]);
  }
  pdl_wait();      // x and the residual belong to the step: nothing of them is touched above this line
  pdl_trigger();
#pragma unroll
  for (int s = 0; s < PRE; s++) dl_ask_x16<T, NT>(p, s < per ? k0 + s * kDlRows : p.k, x[s]);
  if constexpr (LN) dl_ln_stats<T, LN>(p, st);
  float acc[NT][4][4];
  dl_zero<NT>(acc);
#pragma unroll
  for (int s = 0; s < PRE; s++) dl_products16<T, NT, LN != 0>(wv[s], x[s], gam[s], bet[s], st, acc);
  for (int s = PRE; s < per; s++) {
    dl_load_weights<T>(p, n0, k0 + s * kDlRows, wv[0]);
    dl_ask_x16<T, NT>(p, k0 + s * kDlRows, x[0]);
    if constexpr (LN) dl_ask_norm16<T>(p, k0 + s * kDlRows, gam[0], bet[0]);
    dl_products16<T, NT, LN != 0>(wv[0], x[0], gam[0], bet[0], st, acc);
  }
  if constexpr (LN) dl_unit<T, NT>(acc);
  dl_store16<NT>(acc, sSum[threadIdx.x >> 5]);
  __syncthreads();
  dl_finish<T, NT * 8>(p, n0, rank, ranks, &sSum[0][0][0], sFin);
}

// ── a layer's QKV projection and its attention in one launch (16-bit weights) ─
// A cluster of eight CTAs has one head. Its first CTAs take the shares of K of the head's 192 columns, with the loads, the layer_norm and
// the order of additions of decode_linear_kernel; instead of going to memory as q | k | v their sums go to the CTAs that attend, one
// sequence each, whose cached rows were asked for before the dependency wait. That takes the place of a launch and of the round trip of
// q | k | v through the L2: 8.6 us for the two, 7.5 for this; GPT-2 small, 64 + 50 tokens of eight sequences in bf16, 14.6 -> 13.55 ms, a step
// of one sequence 221 -> 218 us. (Cached rows asked for behind the products: no gain. Two sequences a CTA for batches of up to sixteen 383 -> 393 us a
// step; with 160 or 256 clusters' CTAs, more than SMs, at width 1280 245 -> 280 and at 2048 291 -> 322.)
constexpr int kDqRanks = 8, kDqCols = 3 * kDlCols;
struct DecodeAttnParams { void* kcache; void* vcache; void* out; const int* len_ptr; int heads, t_max; float scale; };
constexpr int kDqSums = 3 * (kDlThreads / 32) * kDqRanks * kDlSumPitch, kDqFin = kDqRanks * kDqCols;      // floats
template <typename T>
__global__ void __launch_bounds__(kDlThreads) decode_qkv_attention_kernel(const __grid_constant__ DecodeLinearParams p, const __grid_constant__ DecodeAttnParams a, int shares) {
  extern __shared__ __align__(16) float dq_smem[];
  constexpr int W = kDlThreads / 32, ROWS = kDqRanks;
  float* const sSum = dq_smem;                             // [q, k, v][warp][row][column]
  float* const sFin = sSum + kDqSums;                      // [share][column] of this CTA's sequence
  float* const s_scores = sFin + kDqFin;                   // [t_max]
  __shared__ DlStats st;
  __shared__ AttnDecodeSmem sm;
  __shared__ float s_qkv[kDqCols];
  const int rank = (int)sm100::cluster_ctarank(), h = blockIdx.x, d = a.heads * 64, tid = threadIdx.x, warp = tid >> 5;
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  const bool works = rank < shares, attends = rank < p.m;
  const int k0 = rank * kDlRows;                           // a slab a share
  uint4 wv[3][4];
  uint2 x[1], gam = make_uint2(0u, 0u), bet = gam;
  if (works) {
#pragma unroll
    for (int c = 0; c < 3; c++) dl_load_weights<T>(p, c * d + h * 64, k0, wv[c]);
    dl_ask_norm16<T>(p, k0, gam, bet);
  }
  float bias = 0.f;
  if (tid < kDqCols && p.bias) bias = Cvt<T>::to(reinterpret_cast<const T*>(p.bias)[(tid >> 6) * d + h * 64 + (tid & 63)]);
  const int len = attn_decode_len(*a.len_ptr, a.t_max);    // older than the launch before this one, as are the cached rows below it (attention_decode_kernel)
  AttnDecodeRegs<T> pre;
  const long long at_head = ((long long)rank * a.heads + h) * (long long)a.t_max * 64;
  T* const kc = reinterpret_cast<T*>(a.kcache) + at_head;
  T* const vc = reinterpret_cast<T*>(a.vcache) + at_head;
  if (attends) attn_decode_fetch<T>(kc, vc, len, pre);
  pdl_wait();      // x belongs to the step
  pdl_trigger();
  if (works) {
    dl_ask_x16<T, 1>(p, k0, x);
    dl_ln_stats<T, 4>(p, st);
#pragma unroll
    for (int c = 0; c < 3; c++) {
      float acc[1][4][4];
      dl_zero<1>(acc);
      dl_products16<T, 1, true>(wv[c], x, gam, bet, st, acc);
      dl_unit<T, 1>(acc);
      dl_store16<1>(acc, reinterpret_cast<float (*)[kDlSumPitch]>(sSum + (c * W + warp) * ROWS * kDlSumPitch));
    }
  }
  __syncthreads();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (works) {
    for (int i = tid; i < p.m * kDqCols; i += kDlThreads) {
      const int m = i / kDqCols, c = i - m * kDqCols;
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < W; w++) v += sSum[(((c >> 6) * W + w) * ROWS + m) * kDlSumPitch + (c & 63)];      // warp order = K order
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(sm100::mapa_u32(sm100::smem_u32(sFin + rank * kDqCols + c), (uint32_t)m)), "f"(v) : "memory");
    }
  }
  sm100::cluster_sync_all();
  if (!attends) return;
  if (tid < kDqCols) {
    float v = 0.f;
    for (int r = 0; r < shares; r++) v += sFin[r * kDqCols + tid];
    s_qkv[tid] = Cvt<T>::to(Cvt<T>::from(v + bias));
  }
  __syncthreads();
  attn_decode_item<T>(s_qkv, kc, vc, reinterpret_cast<T*>(a.out) + (long long)rank * d + h * 64, len, a.scale, s_scores, sm, pre);
}

// float32 weights: the same on CUDA cores, x staged in shared memory; ROWS of it, eight or sixteen. The slabs of a share behind the first are
// on their way to the L2 before the dependency wait. A step of GPT-2 small with 1 / 8 / 16 sequences, us: 463 / 579 / 793 with a CTA per
// slab and partial sums in the L2, 518 / 590 / 780 with clusters and sixteen rows for any batch, now 372 / 444 / 808 (a box
// 2 % slower); four layers of width 2048: 663 / 755 / 1 258, 719 / 812 / 1 303, now 619 / 677 / 1 178.
template <int ROWS, bool LN>
__global__ void __launch_bounds__(kDlThreads) decode_linear_f32_kernel(const __grid_constant__ DecodeLinearParams p, int per) {
  __shared__ __align__(16) float sSum[kDlThreads / 32][ROWS][kDlSumPitch];
  __shared__ __align__(16) float sBuf[ROWS * (kDlRows + kDlXPad)];       // x, then the shares' sums
  static_assert((ROWS + kDlShares) * kDlCols <= ROWS * (kDlRows + kDlXPad), "the shares' sums take the place of x");
  __shared__ DlStats st;
  const int ranks = gridDim.y, rank = ranks > 1 ? (int)sm100::cluster_ctarank() : 0;
  const int n0 = blockIdx.x * kDlCols, k0 = rank * per * kDlRows;
  uint4 wv[8];
  DlX<float> x;
  dl_load_weights<float>(p, n0, k0, wv);
  if constexpr (LN) dl_ask_norm<float>(p, k0, x);
  for (int s = 1; s < per; s++) {                          // 256 bytes of each of 128 rows
    const int kk = k0 + s * kDlRows + (threadIdx.x >> 1), col = n0 + (threadIdx.x & 1) * 32;
    if (kk < p.k && col < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const float*>(p.w) + (long long)kk * p.w_row + col));
  }
  pdl_wait();
  pdl_trigger();
  dl_ask_x<float>(p, k0, x);
  if constexpr (LN) dl_ln_stats<float>(p, st);
  float acc[ROWS][4];
#pragma unroll
  for (int m = 0; m < ROWS; m++) { acc[m][0] = 0.f; acc[m][1] = 0.f; acc[m][2] = 0.f; acc[m][3] = 0.f; }
  for (int s = 0; s < per; s++) {
    if (s) {
      __syncthreads();
      dl_load_weights<float>(p, n0, k0 + s * kDlRows, wv);
      if constexpr (LN) dl_ask_norm<float>(p, k0 + s * kDlRows, x);
      dl_ask_x<float>(p, k0 + s * kDlRows, x);
    }
    dl_put_x<float, ROWS, LN>(p, st, sBuf, kDlRows + kDlXPad, k0 + s * kDlRows, x);
    __syncthreads();
    dl_products_f32(sBuf, kDlRows + kDlXPad, wv, acc);
  }
  dl_store_f32(acc, sSum);
  __syncthreads();
  if (ranks > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");     // every CTA is done with its x
  dl_finish<float, ROWS>(p, n0, rank, ranks, &sSum[0][0][0], sBuf);
}


bool decode_linear_eligible(const GemmDesc& d) {
  if (!(d.dtype == DType::BF16 || d.dtype == DType::F16 || d.dtype == DType::F32) || d.b_dtype != d.dtype) return false;
  if (d.c_f32 || d.ep.argmax_keys || d.ep.b_scales || d.ep.alpha != 1.0f) return false;
  if (d.batch != 1 || d.batch_inner != 1 || d.m < 1 || d.m > kDlMaxM || d.n < 64 || d.n > 65536 || d.k < 16) return false;
  if (d.a_col != 1 || d.b_col != 1 || d.b_row % 4 != 0 || d.n % 4 != 0) return false;      // W stored [K, N]; 4-element loads
  const uintptr_t align = d.dtype == DType::F32 ? 15u : 7u;
  if ((reinterpret_cast<uintptr_t>(d.b) & align) != 0) return false;
  const int n16 = d.dtype == DType::F32 ? 4 : 8;
  if (d.a_row % n16 != 0 || (reinterpret_cast<uintptr_t>(d.a) & 15u) != 0 || d.k % 8 != 0) return false;   // 16-byte loads of x
  if (d.ln_gamma && (d.k % n16 != 0 || d.k > 256 * n16)) return false;                                     // a row fits the registers of one warp
  const int64_t ks = (d.k + kDlRows - 1) / kDlRows;
  return ks <= 64;
}

template <typename K>
static cudaError_t launch_dl(cudaStream_t s, K kernel, const DecodeLinearParams& p, int per, int ranks) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.n + kDlCols - 1) / kDlCols), (unsigned)ranks); cfg.blockDim = dim3(kDlThreads); cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = (unsigned)ranks; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = ranks > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, p, per);
}
template <typename T, int NT>
static cudaError_t launch_dl16(cudaStream_t s, const DecodeLinearParams& p, int per, int ranks) {
  if (!p.ln_gamma) return per == 1 ? launch_dl(s, decode_linear_kernel<T, NT, 1, 0>, p, per, ranks) : launch_dl(s, decode_linear_kernel<T, NT, 3, 0>, p, per, ranks);
  return p.k <= 1024 ? launch_dl(s, decode_linear_kernel<T, NT, 1, 4>, p, per, ranks) : launch_dl(s, decode_linear_kernel<T, NT, 1, 8>, p, per, ranks);
}

template <int ROWS>
static cudaError_t launch_dl_f32(cudaStream_t s, const DecodeLinearParams& p, int per, int ranks) {
  return p.ln_gamma ? launch_dl(s, decode_linear_f32_kernel<ROWS, true>, p, per, ranks) : launch_dl(s, decode_linear_f32_kernel<ROWS, false>, p, per, ranks);
}

Status decode_linear(cudaStream_t s, const GemmDesc& d) {
  if (!decode_linear_eligible(d)) return Status::invalid("decode_linear: shape or layout not supported");
  DecodeLinearParams p;
  p.x = d.a; p.w = d.b; p.y = d.c; p.bias = d.ep.bias; p.residual = d.ep.residual; p.ln_gamma = d.ln_gamma; p.ln_beta = d.ln_beta; p.ln_eps = d.ln_eps;
  p.act = (int)d.ep.act; p.m = (int)d.m; p.n = (int)d.n; p.k = (int)d.k;
  p.x_row = d.a_row; p.w_row = d.b_row; p.y_row = d.c_row; p.partial = nullptr;
  const int per = dl_per((int)((d.k + kDlRows - 1) / kDlRows)), ranks = dl_shares((int)d.k);
  cudaError_t e;
  if (d.dtype == DType::F32) e = d.m <= 8 ? launch_dl_f32<8>(s, p, per, ranks) : launch_dl_f32<16>(s, p, per, ranks);
  else if (d.dtype == DType::BF16) e = d.m <= 8 ? launch_dl16<__nv_bfloat16, 1>(s, p, per, ranks) : launch_dl16<__nv_bfloat16, 2>(s, p, per, ranks);
  else e = d.m <= 8 ? launch_dl16<__half, 1>(s, p, per, ranks) : launch_dl16<__half, 2>(s, p, per, ranks);
  return cuda_status(e, "decode_linear");
}

// At most eight sequences (a cluster has one CTA for each), more than four shares of K (nine heads: with fewer the two launches have clusters
// of at most four), and no more clusters than run at once with one CTA an SM (238 registers): two thirds of the SMs, as clusters of eight do
// not fill every group of SMs; with 148 SMs that is twelve heads. A step of six layers, us, two launches / one:
//   heads      1          4          8          9          10         11         12         13         14         15         16
//   1 seq.,    64 rows    70 / 74    82 / 86    97 / 100   105 / 101  107 / 102  111 / 111  113 / 111  132 / 131  135 / 138  148 / 148  149 / 167
//   8 seq.,    64 rows    78 / 84    94 / 96    110 / 113  117 / 110  120 / 111  127 / 127  130 / 119  156 / 150  159 / 159  178 / 172  182 / 205
//   8 seq.,   900 rows    114 / 122  129 / 133  171 / 178  189 / 183  193 / 186  199 / 197  201 / 200  225 / 220  229 / 228  246 / 243  249 / 334
// and eight behind 7 900 rows 615 / 600 with twelve heads, 597 / 587 with nine. Thirteen to fifteen differ by -4 to +2 % and stay apart.
bool decode_qkv_attention_eligible(const GemmDesc& d, int heads, int t_max) {
  return d.dtype != DType::F32 && d.ln_gamma && decode_linear_eligible(d) && d.k == heads * 64 && d.k > 4 * kDlRows && d.k <= kDqRanks * kDlRows /* a slab a share */ &&
         d.n == 3 * d.k && d.m <= kDqRanks && heads * kDqRanks * 3 <= sm_count() * 2 && !d.ep.residual && d.ep.act == Act::None && t_max >= 1 && t_max <= 8192;
}
template <typename T>
static cudaError_t launch_dq(cudaStream_t s, const DecodeLinearParams& p, const DecodeAttnParams& a, int shares) {
  constexpr int fixed = (kDqSums + kDqFin) * (int)sizeof(float);
  static bool attr = false;
  if (!attr) {
    const cudaError_t e = cudaFuncSetAttribute(decode_qkv_attention_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, fixed + 8192 * (int)sizeof(float));
    if (e != cudaSuccess) return e;
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)a.heads, kDqRanks); cfg.blockDim = dim3(kDlThreads); cfg.stream = s; cfg.dynamicSmemBytes = (size_t)fixed + a.t_max * sizeof(float);
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = 1; at[1].val.clusterDim.y = kDqRanks; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, decode_qkv_attention_kernel<T>, p, a, shares);
}
Status decode_qkv_attention(cudaStream_t s, const GemmDesc& d, void* kcache, void* vcache, void* out, const int* len_ptr, int heads, int t_max, float scale) {
  if (!decode_qkv_attention_eligible(d, heads, t_max)) return Status::invalid("decode_qkv_attention: shape or layout not supported");
  if (!aligned16(kcache) || !aligned16(vcache)) return Status::compute("decode_qkv_attention needs 16-byte aligned caches");
  DecodeLinearParams p;
  p.x = d.a; p.w = d.b; p.y = nullptr; p.bias = d.ep.bias; p.residual = nullptr; p.ln_gamma = d.ln_gamma; p.ln_beta = d.ln_beta; p.ln_eps = d.ln_eps;
  p.act = (int)Act::None; p.m = (int)d.m; p.n = (int)d.n; p.k = (int)d.k;
  p.x_row = d.a_row; p.w_row = d.b_row; p.y_row = 0; p.partial = nullptr;
  DecodeAttnParams a{kcache, vcache, out, len_ptr, heads, t_max, scale};
  const int shares = dl_shares((int)d.k);
  const cudaError_t e = d.dtype == DType::BF16 ? launch_dq<__nv_bfloat16>(s, p, a, shares) : launch_dq<__half>(s, p, a, shares);
  return cuda_status(e, "decode_qkv_attention");
}

// ── the tied LM head of a step with its greedy pick ─────────────────────────
// x [m, k] against the embedding [vocab, k], both K-major, m <= 16: bound by reading the embedding once. A warp has 16 of its rows, which are
// the rows of mma.m16n8k16, over the whole of K, straight from memory (the order of K inside a block of 32 columns is free, so a lane feeds
// two products from one 16-byte piece of either operand); what is asked for first is on its way ahead of the dependency wait. The pick is that of
// the matrix product's argmax epilogue: values as they would be stored, the lowest column among equals, a NaN in column 0 kept. A warp
// looks at the keys before it touches them, so that thousands of warps do not queue for one line.
// GPT-2 small, eight sequences, bf16: 21.7 us a launch with 128 x 192 tiles on tcgen05, 15.3 with this (77 MB).
constexpr int kDhWarps = 4;
__device__ __forceinline__ unsigned long long dh_key(float r, int col) {
  if (r != r) return col == 0 ? 0xffffffffffffffffull : 0ull;
  const uint32_t b = __float_as_uint(r), ord = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  return ((unsigned long long)ord << 32) | (unsigned long long)(0xffffffffu - (uint32_t)col);
}
template <typename T, int NT>        // NT groups of eight rows of x
__global__ void __launch_bounds__(kDhWarps * 32) decode_head_kernel(const T* __restrict__ w, const T* __restrict__ x, unsigned long long* keys, int m, int vocab, int k) {
  constexpr int U = 4;               // blocks of 32 columns in flight
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3, n0 = (blockIdx.x * kDhWarps + (threadIdx.x >> 5)) * 16;
  if (n0 >= vocab) return;
  const T* w0 = w + (long long)min(n0 + g, vocab - 1) * k + q * 8;
  const T* w1 = w + (long long)min(n0 + g + 8, vocab - 1) * k + q * 8;
  uint4 a0[U], a1[U];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (c0 + u * 32 >= k) break;
      a0[u] = __ldcs(reinterpret_cast<const uint4*>(w0 + c0 + u * 32)); a1[u] = __ldcs(reinterpret_cast<const uint4*>(w1 + c0 + u * 32));
    }
  };
  fetch(0);
  pdl_wait();
  pdl_trigger();
  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; t++) { acc[t][0] = 0.f; acc[t][1] = 0.f; acc[t][2] = 0.f; acc[t][3] = 0.f; }
  for (int c0 = 0; c0 < k; c0 += U * 32) {
    uint4 b[U][NT];
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int t = 0; t < NT; t++)
        b[u][t] = c0 + u * 32 < k && g + 8 * t < m ? *reinterpret_cast<const uint4*>(x + (long long)(g + 8 * t) * k + c0 + u * 32 + q * 8) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (c0 + u * 32 >= k) break;
#pragma unroll
      for (int t = 0; t < NT; t++) {
        mma_16816<T>(acc[t], a0[u].x, a1[u].x, a0[u].y, a1[u].y, b[u][t].x, b[u][t].y);
        mma_16816<T>(acc[t], a0[u].z, a1[u].z, a0[u].w, a1[u].w, b[u][t].z, b[u][t].w);
      }
    }
    if (c0 + U * 32 < k) fetch(c0 + U * 32);
  }
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int j = 0; j < 2; j++) {    // this lane: embedding rows g and g + 8 for row 2 q + j of x
      unsigned long long key = 0ull;
      if (n0 + g < vocab) key = dh_key(Cvt<T>::to(Cvt<T>::from(acc[t][j])), n0 + g);
      if (n0 + g + 8 < vocab) { const unsigned long long o = dh_key(Cvt<T>::to(Cvt<T>::from(acc[t][2 + j])), n0 + g + 8); key = o > key ? o : key; }
#pragma unroll
      for (int d = 4; d < 32; d *= 2) { const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, d); key = o > key ? o : key; }
      const int row = t * 8 + 2 * q + j;
      if (g == 0 && row < m && key > *reinterpret_cast<volatile unsigned long long*>(keys + row)) atomicMax(keys + row, key);
    }
}
bool decode_head_eligible(DType dt, const void* w, const void* x, int m, int64_t k) {
  return (dt == DType::BF16 || dt == DType::F16) && m >= 1 && m <= 16 && k >= 32 && k % 32 == 0 && k <= 65536 && aligned16(w) && aligned16(x);
}
Status decode_head(cudaStream_t s, DType dt, const void* w, const void* x, unsigned long long* keys, int m, int vocab, int k) {
  if (!decode_head_eligible(dt, w, x, m, k) || vocab < 1) return Status::invalid("decode_head: shape or layout not supported");
  const dim3 grid((unsigned)((vocab + 16 * kDhWarps - 1) / (16 * kDhWarps))), block(kDhWarps * 32);
#define AG_DH(T) (m <= 8 ? launch_pdl(decode_head_kernel<T, 1>, grid, block, 0, s, (const T*)w, (const T*)x, keys, m, vocab, k) \
                         : launch_pdl(decode_head_kernel<T, 2>, grid, block, 0, s, (const T*)w, (const T*)x, keys, m, vocab, k))
  const cudaError_t e = dt == DType::BF16 ? AG_DH(__nv_bfloat16) : AG_DH(__half);
#undef AG_DH
  return cuda_status(e, "decode_head");
}

// ── the layers of a decode step as one persistent kernel ────────────────────
// Sixty dependent launches of a few microseconds each have their drain, dependency resolution and ramp in between (a trivial launch
// takes 1.8 µs inside a CUDA graph with programmatic edges). Here one cooperative grid walks all layers and separates the phases with a grid-wide barrier of its own (~1 µs):
//   E    x = wte[tok] + wpe[pos]
//   per layer:
//   P1   partial products of ln_1(x) @ W_qkv                      (36 x 6 items of 64 columns x 128 K rows)
//   P2   attention per (sequence, head): q, k, v summed from P1's partials, cache appended in place   (B x heads items)
//   P3   partial products of att @ W_proj                         (12 x 6 items)
//   P3b  x2 = x + sum of P3's partials + bias                     (element-wise)
//   P4   partial products of ln_2(x2) @ W_fc                      (48 x 6 items)
//   P5   partial products of gelu(P4 + bias) @ W_fc2, the operand summed from P4's partials on the way in   (12 x 8 items)
//   P5b  x = x2 + sum of P5's partials + bias                     (element-wise)
// Every item runs the same device functions, in the same order of additions, as the per-op kernels above, so the
// stream of tokens is the one the per-op engine produces. The barrier: one counter in global memory, cleared by a
// memset node before the launch; each CTA adds one and spins (bounded: 2 s, then an error word is set and every CTA
// leaves at its next barrier) until the count reaches phases-so-far x CTAs. The launch is cooperative, so all CTAs
// are resident and the spin cannot wait for a CTA that has not started.
constexpr int kMegaCols = 2048;      // of a row at most: what the statistics of layer_norm keep in registers
struct MegaLayerW {
  const void *ln1_g, *ln1_b, *w_qkv, *b_qkv, *w_proj, *b_proj, *ln2_g, *ln2_b, *w_fc, *b_fc, *w_fc2, *b_fc2;
  void *kcache, *vcache;
};
struct MegaParams {
  const MegaLayerW* layers;
  int n_layer, heads, d, t_max, batch;
  const void *wte, *wpe;
  const int32_t *tok, *pos;
  const int* len_ptr;
  void *x, *x2, *att;             // [16][d] of the storage type
  float* partial;                 // four regions: qkv, proj, fc, fc2 partials
  unsigned int* bar;
  int* err;
  float scale;
};

#ifdef AG_DECODE_PROBE
__device__ unsigned long long g_mega_probe[2048];   // CTA 0: time after every barrier (ns)
__device__ int g_mega_probe_n;
#endif
__device__ __forceinline__ bool mega_barrier(const MegaParams& p, unsigned int& target) {
#ifdef AG_DECODE_PROBE
  if (blockIdx.x == 0 && threadIdx.x == 0 && g_mega_probe_n < 2046) g_mega_probe[g_mega_probe_n++] = globaltimer_ns_dec();   // arrival
#endif
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(p.bar, 1u);
    const unsigned long long t0 = globaltimer_ns_dec();
    unsigned int spins = 0;
    while (true) {
      unsigned int seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.bar) : "memory");
      if (seen >= target) break;
      if ((++spins & 0x3ffu) == 0) {
        if (*reinterpret_cast<volatile int*>(p.err) != 0) break;
        if (globaltimer_ns_dec() - t0 > 2000000000ull) { atomicCAS(p.err, 0, 31); break; }
      }
    }
    __threadfence();
  }
  __syncthreads();
#ifdef AG_DECODE_PROBE
  if (blockIdx.x == 0 && threadIdx.x == 0 && g_mega_probe_n < 2046) g_mega_probe[g_mega_probe_n++] = globaltimer_ns_dec();   // release
#endif
  return *reinterpret_cast<volatile int*>(p.err) == 0;
}

template <typename T>
__global__ void __launch_bounds__(kDlThreads, 2) decode_layers_kernel(const MegaParams p) {
#ifdef AG_DECODE_PROBE
  if (blockIdx.x == 0 && threadIdx.x == 0) { g_mega_probe_n = 0; g_mega_probe[g_mega_probe_n++] = globaltimer_ns_dec(); }
#endif
  extern __shared__ float s_scores[];          // [t_max]
  __shared__ DlSmem sm;
  __shared__ AttnDecodeSmem asm_;
  __shared__ float s_qkv[192];
  const int D = p.d, B = p.batch;
  const int G = (int)gridDim.x, cta = (int)blockIdx.x;
  unsigned int target = 0;
  float* part_qkv = p.partial;
  const int ks_d = dl_shares(D), ks_4d = dl_shares(4 * D);
  float* part_proj = part_qkv + (long long)ks_d * kDlMaxM * 3 * D;
  float* part_fc = part_proj + (long long)ks_d * kDlMaxM * D;
  float* part_fc2 = part_fc + (long long)ks_d * kDlMaxM * 4 * D;

  // The weights of this CTA's first item of the next linear phase are fetched as soon as the current linear phase is
  // done (they are constants of the model): the loads fly during the barriers and the phases in between, as the per-op
  // kernels fetch theirs ahead of the dependency wait.
  uint4 wv_next[kDlWv<T>];
  auto prefetch = [&](const void* wgt, int n, int k) {
    DecodeLinearParams lp{};
    lp.w = wgt; lp.n = n; lp.k = k; lp.w_row = n;
    const int n_slabs = (n + kDlCols - 1) / kDlCols, shares = dl_shares(k), per = dl_per((k + kDlRows - 1) / kDlRows);
    if (cta < n_slabs * shares) dl_load_weights<T>(lp, (cta % n_slabs) * kDlCols, (cta / n_slabs) * per * kDlRows, wv_next);
  };
  // one linear's partial products over the grid
  auto linear_partials = [&](DecodeLinearParams lp) {
    const int n_slabs = (lp.n + kDlCols - 1) / kDlCols, shares = dl_shares(lp.k), per = dl_per((lp.k + kDlRows - 1) / kDlRows);
    bool stats = false;
    for (int it = cta; it < n_slabs * shares; it += G) {
      const int ns = it % n_slabs, ks = it / n_slabs;
      uint4 wv[kDlWv<T>];
      if (it == cta) {
#pragma unroll
        for (int i = 0; i < kDlWv<T>; i++) wv[i] = wv_next[i];
      } else {
        dl_load_weights<T>(lp, ns * kDlCols, ks * per * kDlRows, wv);
      }
      __syncthreads();                       // the previous item's shared-memory reads are done
      if (lp.ln_gamma && !stats) { dl_ln_stats<T, kMegaCols / (32 * Pack<T>::N)>(lp, sm.st); stats = true; }
      dl_partial<T>(lp, sm, ns * kDlCols, ks, per, wv);
    }
  };
  // y = round(sum of partials + bias + residual) over the grid
  auto finish_rows = [&](const DecodeLinearParams& lp, int shares) {
    T* Y = reinterpret_cast<T*>(lp.y);
    for (int i = cta * kDlThreads + threadIdx.x; i < lp.m * lp.n; i += G * kDlThreads) {
      const int m = i / lp.n, c = i % lp.n;
      Y[(long long)m * lp.y_row + c] = Cvt<T>::from(dl_finish_element<T>(lp, shares, m, c));
    }
  };

  // E: embeddings (a row per CTA; the sum rounded once, as the embedding kernel stores it)
  for (int b = cta; b < B; b += G) {
    const T* te = reinterpret_cast<const T*>(p.wte) + (long long)p.tok[b] * D;
    const T* pe = reinterpret_cast<const T*>(p.wpe) + (long long)p.pos[b] * D;
    T* xr = reinterpret_cast<T*>(p.x) + (long long)b * D;
    for (int i = threadIdx.x; i < D; i += kDlThreads) xr[i] = Cvt<T>::from(Cvt<T>::to(te[i]) + Cvt<T>::to(pe[i]));
  }
  prefetch(p.layers[0].w_qkv, 3 * D, D);
  if (!mega_barrier(p, target)) return;

  for (int l = 0; l < p.n_layer; l++) {
    const MegaLayerW& w = p.layers[l];
    DecodeLinearParams lp;
    // P1: ln_1(x) @ W_qkv
    lp = DecodeLinearParams{};
    lp.x = p.x; lp.w = w.w_qkv; lp.ln_gamma = w.ln1_g; lp.ln_beta = w.ln1_b; lp.ln_eps = 1e-5f;
    lp.m = B; lp.n = 3 * D; lp.k = D; lp.x_row = D; lp.w_row = 3 * D; lp.y_row = 3 * D; lp.partial = part_qkv;
    linear_partials(lp);
    prefetch(w.w_proj, D, D);
    if (!mega_barrier(p, target)) return;
    // P2: attention; q | k | v of the new token = P1's partials + bias, rounded as the projection would have stored them
    for (int it = cta; it < B * p.heads; it += G) {
      const int b = it / p.heads, h = it % p.heads;
      __syncthreads();
      for (int i = threadIdx.x; i < 192; i += kDlThreads) {
        const int col = (i >> 6) * D + h * 64 + (i & 63);
        float t = 0.f;
        for (int ks = 0; ks < ks_d; ks++) t += __ldcg(part_qkv + ((long long)ks * kDlMaxM + b) * 3 * D + col);
        t += Cvt<T>::to(reinterpret_cast<const T*>(w.b_qkv)[col]);
        s_qkv[i] = Cvt<T>::to(Cvt<T>::from(t));
      }
      __syncthreads();
      T* kc = reinterpret_cast<T*>(w.kcache) + ((long long)b * p.heads + h) * (long long)p.t_max * 64;
      T* vc = reinterpret_cast<T*>(w.vcache) + ((long long)b * p.heads + h) * (long long)p.t_max * 64;
      const int len = attn_decode_len(*p.len_ptr, p.t_max);
      AttnDecodeRegs<T> pre;
      attn_decode_fetch<T>(kc, vc, len, pre);
      attn_decode_item<T>(s_qkv, kc, vc, reinterpret_cast<T*>(p.att) + (long long)b * D + h * 64, len, p.scale, s_scores, asm_, pre);
    }
    if (!mega_barrier(p, target)) return;
    // P3: att @ W_proj, then x2 = x + that + bias
    lp = DecodeLinearParams{};
    lp.x = p.att; lp.w = w.w_proj; lp.m = B; lp.n = D; lp.k = D; lp.x_row = D; lp.w_row = D; lp.y_row = D; lp.partial = part_proj;
    linear_partials(lp);
    prefetch(w.w_fc, 4 * D, D);
    if (!mega_barrier(p, target)) return;
    lp.y = p.x2; lp.bias = w.b_proj; lp.residual = p.x;
    finish_rows(lp, ks_d);
    if (!mega_barrier(p, target)) return;
    // P4: ln_2(x2) @ W_fc
    lp = DecodeLinearParams{};
    lp.x = p.x2; lp.w = w.w_fc; lp.ln_gamma = w.ln2_g; lp.ln_beta = w.ln2_b; lp.ln_eps = 1e-5f;
    lp.m = B; lp.n = 4 * D; lp.k = D; lp.x_row = D; lp.w_row = 4 * D; lp.y_row = 4 * D; lp.partial = part_fc;
    linear_partials(lp);
    prefetch(w.w_fc2, D, 4 * D);
    if (!mega_barrier(p, target)) return;
    // P5: gelu(P4 + bias) @ W_fc2, then x = x2 + that + bias
    lp = DecodeLinearParams{};
    lp.x = nullptr; lp.xp = part_fc; lp.xp_shares = ks_d; lp.xp_bias = w.b_fc; lp.xp_act = (int)Act::GeluTanh;
    lp.w = w.w_fc2; lp.m = B; lp.n = D; lp.k = 4 * D; lp.x_row = 4 * D; lp.w_row = D; lp.y_row = D; lp.partial = part_fc2;
    linear_partials(lp);
    if (l + 1 < p.n_layer) prefetch(p.layers[l + 1].w_qkv, 3 * D, D);
    if (!mega_barrier(p, target)) return;
    lp.y = p.x; lp.bias = w.b_fc2; lp.residual = p.x2;
    finish_rows(lp, ks_4d);
    if (!mega_barrier(p, target)) return;
  }
}

// Enqueues the barrier reset and the cooperative launch. `layers` is a device array of n_layer entries.
Status decode_layers(cudaStream_t s, DType dt, const void* layers, int n_layer, int heads, int d, int t_max, int batch, const void* wte, const void* wpe,
                     const int32_t* tok, const int32_t* pos, const int* len_ptr, void* x, void* x2, void* att, unsigned int* bar, int* err) {
  if (batch < 1 || batch > kDlMaxM || d != heads * 64 || d % 8 != 0 || t_max < 1 || t_max > 8192) return Status::invalid("decode_layers: shape not supported");
  if (d > kMegaCols) return Status::unsupported("decode_layers: rows of more than " + std::to_string(kMegaCols) + " columns");
  float* partial = skinny_partials();
  if (!partial) return Status::compute("decode_layers: the kernel workspace is not initialised");
  const long long ks_d = dl_shares(d), ks_4d = dl_shares(4 * d);
  const long long need = (ks_d * kDlMaxM * 3 * d) + (ks_d * kDlMaxM * d) + (ks_d * kDlMaxM * 4 * d) + (ks_4d * kDlMaxM * d);
  if (need > ((long long)1 << 18) * 16) return Status::invalid("decode_layers: the partial sums do not fit the workspace");
  MegaParams p;
  p.layers = static_cast<const MegaLayerW*>(layers); p.n_layer = n_layer; p.heads = heads; p.d = d; p.t_max = t_max; p.batch = batch;
  p.wte = wte; p.wpe = wpe; p.tok = tok; p.pos = pos; p.len_ptr = len_ptr; p.x = x; p.x2 = x2; p.att = att;
  p.partial = partial; p.bar = bar; p.err = err; p.scale = 1.0f / sqrtf(64.0f);
  // 47 KB of static shared memory leave next to nothing of the default 48 KB for the scores: longer caches need the opt-in (set
  // on the first, uncaptured call)
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t ae = cudaFuncSetAttribute(decode_layers_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * (int)sizeof(float));
    if (ae == cudaSuccess) ae = cudaFuncSetAttribute(decode_layers_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * (int)sizeof(float));
    if (ae == cudaSuccess) ae = cudaFuncSetAttribute(decode_layers_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8192 * (int)sizeof(float));
    if (ae != cudaSuccess) return cuda_status(ae, "decode_layers shared-memory attribute");
    attr_set = true;
  }
  cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(unsigned int), s);
  if (e != cudaSuccess) return cuda_status(e, "decode_layers barrier reset");
  cudaLaunchConfig_t cfg = {};
  // up to two CTAs per SM (every linear phase then has at most one item per CTA), as many as can be resident together
  int per_sm = 0;
  const size_t dyn = (size_t)t_max * sizeof(float);
  cudaError_t oe = dt == DType::BF16 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_layers_kernel<__nv_bfloat16>, kDlThreads, dyn)
                   : dt == DType::F16 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_layers_kernel<__half>, kDlThreads, dyn)
                                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, decode_layers_kernel<float>, kDlThreads, dyn);
  if (oe != cudaSuccess || per_sm < 1) return Status::compute("decode_layers: the kernel does not fit an SM");
  if (per_sm > 2) per_sm = 2;
  cfg.gridDim = dim3((unsigned)(sm_count() * per_sm), 1, 1);
  cfg.blockDim = dim3(kDlThreads, 1, 1);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  if (dt == DType::BF16) e = cudaLaunchKernelEx(&cfg, decode_layers_kernel<__nv_bfloat16>, p);
  else if (dt == DType::F16) e = cudaLaunchKernelEx(&cfg, decode_layers_kernel<__half>, p);
  else e = cudaLaunchKernelEx(&cfg, decode_layers_kernel<float>, p);
  if (e != cudaSuccess) return cuda_status(e, "decode_layers");
  return Status::OK();
}
#ifdef AG_DECODE_PROBE
extern "C" __attribute__((visibility("default"))) int applegpu_debug_decode_probe(unsigned long long* out, int cap) {
  int n = 0;
  cudaDeviceSynchronize();
  cudaMemcpyFromSymbol(&n, g_mega_probe_n, sizeof(int));
  if (n > cap) n = cap;
  if (n > 0) cudaMemcpyFromSymbol(out, g_mega_probe, sizeof(unsigned long long) * n);
  return n;
}
#endif
size_t decode_layers_table_bytes(int n_layer) { return sizeof(MegaLayerW) * (size_t)n_layer; }
void decode_layers_fill_entry(void* host_table, int l, const void* const* w12, void* kcache, void* vcache) {
  MegaLayerW& e = static_cast<MegaLayerW*>(host_table)[l];
  e.ln1_g = w12[0]; e.ln1_b = w12[1]; e.w_qkv = w12[2]; e.b_qkv = w12[3]; e.w_proj = w12[4]; e.b_proj = w12[5];
  e.ln2_g = w12[6]; e.ln2_b = w12[7]; e.w_fc = w12[8]; e.b_fc = w12[9]; e.w_fc2 = w12[10]; e.b_fc2 = w12[11];
  e.kcache = kcache; e.vcache = vcache;
}

// End of a decode step: the picked tokens go into the history, the next step's position ids are written, and the
// step and length counters advance. One block; every thread reads the counters before thread 0 changes them.
// `keys` non-null: the step's tokens are still the (value, column) keys the LM head's row-argmax epilogue merged; this
// kernel turns them into token ids itself (what argmax_finalize does: no key and the sticky-NaN key both mean column 0)
// and clears them for the next step, which saves the step a launch and a memset.
__global__ void decode_finish_kernel(int32_t* __restrict__ tok, int32_t* __restrict__ history, int32_t* __restrict__ pos_ids, int* step_ptr, int* len_ptr,
                                     int batch, int max_steps, unsigned long long* __restrict__ keys) {
  pdl_wait();
  pdl_trigger();
  const int step = *step_ptr, len = *len_ptr;
  __syncthreads();
  for (int t = threadIdx.x; t < batch; t += blockDim.x) {
    int32_t token;
    if (keys) {
      const unsigned long long k = keys[t];
      token = (k == 0ull || k == 0xffffffffffffffffull) ? 0 : (int32_t)(0xffffffffu - (uint32_t)(k & 0xffffffffu));
      keys[t] = 0ull;
      tok[t] = token;
    } else {
      token = tok[t];
    }
    if (step < max_steps) history[(long long)step * batch + t] = token;
    pos_ids[t] = len + 1;
  }
  if (threadIdx.x == 0) { *step_ptr = step + 1; *len_ptr = len + 1; }
}

Status decode_finish(cudaStream_t s, int32_t* tok, int32_t* history, int32_t* pos_ids, int* step_ptr, int* len_ptr, int batch, int max_steps,
                     unsigned long long* keys) {
  cudaError_t le = launch_pdl(decode_finish_kernel, dim3(1), dim3(128), 0, s, tok, history, pos_ids, step_ptr, len_ptr, batch, max_steps, keys);
  if (le != cudaSuccess) return cuda_status(le, "decode_finish");
  return Status::OK();
}

// counters[0] = step, counters[1] = len; pos_ids[0..batch) = len
__global__ void decode_reset_kernel(int* counters, int32_t* pos_ids, int batch, int len) {
  for (int t = threadIdx.x; t < batch; t += blockDim.x) pos_ids[t] = len;
  if (threadIdx.x == 0) { counters[0] = 0; counters[1] = len; }
}
Status decode_reset(cudaStream_t s, int* counters, int32_t* pos_ids, int batch, int len) {
  decode_reset_kernel<<<1, 128, 0, s>>>(counters, pos_ids, batch, len);
  AG_CHECK_LAUNCH("decode_reset");
  return Status::OK();
}

}}  // namespace ag::k
