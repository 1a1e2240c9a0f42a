// Row reductions: layer_norm, softmax / softmax_causal, argmax, sum/mean, sum_dim, mean_all.
//
// Reference semantics: kernel_templates.rs:1075-1116 (layer_norm: mean, population variance,
// 1/sqrt(var+eps)), :398-430 (softmax), :468-497 (softmax_causal: running max starts at -1e9,
// explicit zeros right of the diagonal, half types round exp() to storage before the divide),
// :500-520 (argmax: strict '>' scan from element 0, int32 result). The reference runs one
// thread per row over three serial passes; here a warp owns a row, keeps it in registers after
// a single 16-byte-vectorised read, reduces with shuffles, and writes once.
#include "common.cuh"
#include "sm100.cuh"
#include "tc_math.cuh"
#include <type_traits>
#include <cstdlib>

namespace ag { namespace k {

int* matmul_status_word();

// ── rows in words and by bulk copies ────────────────────────────────────────
// Two 16-bit floats of one word as a pair of floats, and the larger of each of two words (a number beats NaN).
template <typename T> __device__ __forceinline__ uint64_t widen_word(uint32_t w);
template <> __device__ __forceinline__ uint64_t widen_word<__nv_bfloat16>(uint32_t w) { return pack_f32x2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
template <> __device__ __forceinline__ uint64_t widen_word<__half>(uint32_t w) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
  return pack_f32x2(f.x, f.y);
}
template <typename T> __device__ __forceinline__ uint32_t max_word(uint32_t a, uint32_t b) {
  using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  const T2 m = __hmax2(*reinterpret_cast<const T2*>(&a), *reinterpret_cast<const T2*>(&b));
  return *reinterpret_cast<const uint32_t*>(&m);
}

constexpr int kSmSlots = 4, kSmWarps = 4, kSmMinRowBytes = 512;       // row buffers of a warp, warps of a block
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(sm100::smem_u32(src)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  sm100::mbar_expect_tx(bar, bytes);
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(sm100::smem_u32(dst)), "l"(src), "r"(bytes), "r"(sm100::smem_u32(bar)) : "memory");
}
// A warp's end, one lane: rows that it asked for and will not read (a wait for one of them gave up) have landed, or had as long again each, before
// the block's shared memory goes to another; its results have left.
__device__ __forceinline__ void bulk_leave(uint64_t* bar, int64_t row, int64_t asked, int64_t stride, int slot, uint32_t phase, int* status) {
  for (; row < asked; row += stride) {
    sm100::mbar_wait_limit(&bar[slot], phase, status, 9);
    if (++slot == kSmSlots) { slot = 0; phase ^= 1; }
  }
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// Blocks an SM of such a kernel with `smem` bytes of row buffers each; by_registers is the kernel's own, found once.
template <typename K>
static cudaError_t bulk_ctas(K kern, int smem, int max_row_bytes, int* by_registers, int* per_sm) {
  if (!*by_registers) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmWarps * kSmSlots * max_row_bytes);
    int n = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, kSmWarps * 32, 0);
    if (e != cudaSuccess) return e;
    *by_registers = n < 1 ? 1 : n;
  }
  const int by_smem = 227 * 1024 / (smem + 1024 + (int)sizeof(uint64_t) * kSmWarps * kSmSlots);
  *per_sm = by_smem < 1 ? 1 : by_smem < *by_registers ? by_smem : *by_registers;
  return cudaSuccess;
}

// ── layer_norm ──────────────────────────────────────────────────────────────
// Warp-per-row; ITERS packs per lane cover cols <= 32*ITERS*Pack::N. A persistent grid (a few CTAs per SM) walks the
// rows, and a warp keeps TWO rows in flight: the 16-byte loads of its next row are issued before the reductions of
// the current one, so loads, shuffles and stores of neighbouring rows overlap instead of every warp of the grid
// reading at the same time and then writing at the same time. Rows stay in registers as raw packs (converted
// where used), gamma / beta are fetched once per warp.
template <typename T, int ITERS>
__global__ void __launch_bounds__(256) layer_norm_warp_kernel(const T* __restrict__ in, const T* __restrict__ gamma, const T* __restrict__ beta,
                                                               T* __restrict__ out, int64_t rows, int cols, float eps) {
  constexpr int N = Pack<T>::N;
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  const int packs = cols / N;
  const float inv_cols = 1.0f / (float)cols;
  pdl_wait();
  pdl_trigger();
  constexpr bool kHoist = ITERS <= 4;
  Pack<T> gpk[kHoist ? ITERS : 1], bpk[kHoist ? ITERS : 1];
  if (kHoist) {
#pragma unroll
    for (int it = 0; it < (kHoist ? ITERS : 1); it++) {
      int pk = lane + it * 32;
      if (pk < packs) { gpk[it] = ld16(gamma + pk * N); bpk[it] = ld16(beta + pk * N); }
    }
  }
  const int64_t stride = (int64_t)gridDim.x * warps_per_block;
  int64_t row = (int64_t)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  Pack<T> cur[ITERS], nxt[ITERS];
  if (row < rows) {
#pragma unroll
    for (int it = 0; it < ITERS; it++) { int pk = lane + it * 32; if (pk < packs) cur[it] = ld16_stream(in + row * cols + pk * N); }
  }
  for (; row < rows; row += stride) {
    const int64_t next = row + stride;
    if (next < rows) {
#pragma unroll
      for (int it = 0; it < ITERS; it++) { int pk = lane + it * 32; if (pk < packs) nxt[it] = ld16_stream(in + next * cols + pk * N); }
    }
    float sum = 0.f;
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      if (lane + it * 32 < packs) {
#pragma unroll
        for (int e = 0; e < N; e++) sum += Cvt<T>::to(cur[it].v[e]);
      }
    }
    const float mean = warp_sum(sum) * inv_cols;
    float sq = 0.f;
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      if (lane + it * 32 < packs) {
#pragma unroll
        for (int e = 0; e < N; e++) { float d = Cvt<T>::to(cur[it].v[e]) - mean; sq += d * d; }
      }
    }
    const float var = warp_sum(sq) * inv_cols;
    const float inv_std = 1.0f / sqrtf(var + eps);
    T* y = out + row * cols;
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      int pk = lane + it * 32;
      if (pk < packs) {
        Pack<T> g = kHoist ? gpk[kHoist ? it : 0] : ld16(gamma + pk * N);
        Pack<T> b = kHoist ? bpk[kHoist ? it : 0] : ld16(beta + pk * N);
        Pack<T> o;
        float r[N];
#pragma unroll
        for (int e = 0; e < N; e++) r[e] = Cvt<T>::to(g.v[e]) * (Cvt<T>::to(cur[it].v[e]) - mean) * inv_std + Cvt<T>::to(b.v[e]);
        pack_from_floats<T>(o, r);
        st16(y + pk * N, o);   // the next kernel (a GEMM) reads this from L2: no evict-first hint
      }
    }
#pragma unroll
    for (int it = 0; it < ITERS; it++) cur[it] = nxt[it];
  }
}

// The same for many 16-bit rows of 512 to 2560 bytes that come and go by bulk copies (softmax_bulk_kernel below has the
// pipeline), arithmetic on pairs. Rows in registers against bulk copies, bfloat16, us: 131072 x 768 77.3 / 65.6 (6.1 TB/s), 65536 x 1024
// 68.4 / 51.7 (half of it from the L2), 16384 x 1280 19.6 / 17.3, 32768 x 256 12.6 / 11.9, 8192 x 2048 18.2 / 20.0.
// From how many rows an SM on depends on what the kernel above makes of the row (its registers hold two of them). bfloat16 / float16 at 32, 64,
// 112 and 160 rows an SM, in registers and by copies:
//   256 columns   5.5 5.7  5.7 5.6  7.4 7.2  9.8 9.3     / 4.5 4.5  4.8 4.6  7.3 7.2  9.6 9.4
//   512           4.7 4.6  7.3 6.7  11.1 9.4  14.7 11.9  / 4.7 4.5  7.1 6.9  10.7 9.7  14.3 12.2
//   768           5.9 6.7  8.1 8.5  12.4 11.9  16.5 15.1 / 4.9 5.7  8.0 8.5  12.3 12.2  16.3 16.0
//   1024          8.4 6.8  13.1 10.7  20.2 16.3  27.2 21.5 / 6.3 6.5  9.6 10.4  14.6 15.0  19.5 19.4
//   1280          7.8 7.1  12.6 11.8  19.6 17.1  26.5 22.1 / 9.1 7.3  15.5 12.2  18.9 17.6  25.8 22.8
constexpr int kLnMaxRowBytes = 2560;
template <typename T, int ITERS>
__global__ void __launch_bounds__(kSmWarps * 32) layer_norm_bulk_kernel(const T* __restrict__ in, const T* __restrict__ gamma, const T* __restrict__ beta, T* __restrict__ out, int64_t rows,
                                                                         int cols, float eps, int* status) {
  extern __shared__ __align__(128) uint8_t s_rows[];
  __shared__ uint64_t bars[kSmWarps][kSmSlots];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int packs = cols / 8, row_bytes = cols * 2;
  uint8_t* const mine = s_rows + (size_t)warp * kSmSlots * row_bytes;
  uint64_t* const bar = bars[warp];
  if (lane == 0) {
    for (int i = 0; i < kSmSlots; i++) sm100::mbar_init(&bar[i], 1);
    sm100::mbar_fence_init();
  }
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  const int64_t stride = (int64_t)gridDim.x * kSmWarps, row0 = (int64_t)blockIdx.x * kSmWarps + warp;
  int64_t asked = row0;
  if (lane == 0) {
    for (int i = 0; i < kSmSlots - 1 && asked < rows; i++, asked += stride) bulk_load(mine + i * row_bytes, in + asked * cols, (uint32_t)row_bytes, &bar[i]);
  }
  uint4 g[ITERS], b[ITERS];
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    const int pk = lane + it * 32;
    if (pk < packs) { g[it] = *(reinterpret_cast<const uint4*>(gamma) + pk); b[it] = *(reinterpret_cast<const uint4*>(beta) + pk); }
  }
  const float inv_cols = 1.0f / (float)cols;
  int slot = 0, free_slot = kSmSlots - 1;
  uint32_t phase = 0;
  int64_t row = row0;
  for (; row < rows; row += stride) {
    if (lane == 0 && asked < rows) {
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the free slot's copy out has read it
      bulk_load(mine + free_slot * row_bytes, in + asked * cols, (uint32_t)row_bytes, &bar[free_slot]);
      asked += stride;
    }
    if (!__all_sync(0xffffffffu, sm100::mbar_wait_limit(&bar[slot], phase, status, 9))) break;
    uint4* const at = reinterpret_cast<uint4*>(mine + slot * row_bytes);
    uint4 x[ITERS];
    uint64_t s2 = 0;                                       // the bits of (0.f, 0.f)
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      const int pk = lane + it * 32;
      if (pk >= packs) continue;
      x[it] = at[pk];
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&x[it]);
#pragma unroll
      for (int j = 0; j < 4; j++) s2 = add_f32x2(s2, widen_word<T>(w[j]));
    }
    const float mean = warp_sum(sum_f32x2(s2)) * inv_cols;
    const uint64_t nm = pack_f32x2(-mean, -mean);
    uint64_t q2 = 0;
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      if (lane + it * 32 >= packs) continue;
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&x[it]);
#pragma unroll
      for (int j = 0; j < 4; j++) { const uint64_t d = add_f32x2(widen_word<T>(w[j]), nm); q2 = fma_f32x2(d, d, q2); }
    }
    const float inv_std = 1.0f / sqrtf(warp_sum(sum_f32x2(q2)) * inv_cols + eps);
    const uint64_t is = pack_f32x2(inv_std, inv_std);
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      const int pk = lane + it * 32;
      if (pk >= packs) continue;
      const uint32_t *w = reinterpret_cast<const uint32_t*>(&x[it]), *gw = reinterpret_cast<const uint32_t*>(&g[it]), *bw = reinterpret_cast<const uint32_t*>(&b[it]);
      uint4 o;
      uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float lo, hi;
        unpack_f32x2(fma_f32x2(mul_f32x2(widen_word<T>(gw[j]), add_f32x2(widen_word<T>(w[j]), nm)), is, widen_word<T>(bw[j])), lo, hi);
        ow[j] = pack2_t<T>(lo, hi);
      }
      at[pk] = o;
    }
    sm100::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) bulk_store(out + row * cols, at, (uint32_t)row_bytes);
    free_slot = slot;
    if (++slot == kSmSlots) { slot = 0; phase ^= 1; }
  }
  if (lane == 0) bulk_leave(bar, row, asked, stride, slot, phase, status);
}
template <typename T, int ITERS>
static cudaError_t launch_layer_norm_bulk(cudaStream_t s, const T* x, const T* g, const T* b, T* y, int64_t rows, int cols, float eps, int* status) {
  const int smem = kSmWarps * kSmSlots * cols * (int)sizeof(T);
  static int by_registers = 0;
  int per_sm;
  cudaError_t e = bulk_ctas(layer_norm_bulk_kernel<T, ITERS>, smem, kLnMaxRowBytes, &by_registers, &per_sm);
  if (e != cudaSuccess) return e;
  return launch_pdl(layer_norm_bulk_kernel<T, ITERS>, dim3((unsigned)grid_for(rows, kSmWarps, per_sm)), dim3(kSmWarps * 32), (size_t)smem, s, x, g, b, y, rows, cols, eps, status);
}

// Block-per-row, any cols / alignment: three passes over a row that stays in L1/L2.
template <typename T>
__global__ void __launch_bounds__(256) layer_norm_block_kernel(const T* __restrict__ in, const T* __restrict__ gamma, const T* __restrict__ beta,
                                                                T* __restrict__ out, int64_t rows, int64_t cols, float eps) {
  __shared__ float red[33];
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* x = in + row * cols;
    float s = 0.f;
    for (int64_t j = threadIdx.x; j < cols; j += blockDim.x) s += Cvt<T>::to(x[j]);
    float mean = block_sum(s, red) / (float)cols;
    float q = 0.f;
    for (int64_t j = threadIdx.x; j < cols; j += blockDim.x) { float d = Cvt<T>::to(x[j]) - mean; q += d * d; }
    float var = block_sum(q, red) / (float)cols;
    float inv_std = 1.0f / sqrtf(var + eps);
    T* y = out + row * cols;
    for (int64_t j = threadIdx.x; j < cols; j += blockDim.x)
      y[j] = Cvt<T>::from(Cvt<T>::to(gamma[j]) * (Cvt<T>::to(x[j]) - mean) * inv_std + Cvt<T>::to(beta[j]));
  }
}

template <typename T>
static Status layer_norm_t(cudaStream_t s, const TView& in, const TView& gamma, const TView& beta, float eps, const TView& out) {
  constexpr int N = Pack<T>::N;
  int64_t cols = in.shape.back();
  int64_t rows = cols ? in.numel() / cols : 0;
  if (rows == 0 || cols == 0) return Status::OK();
  const T* x = (const T*)in.ptr; const T* g = (const T*)gamma.ptr; const T* b = (const T*)beta.ptr; T* y = (T*)out.ptr;
  bool vec = cols % N == 0 && aligned16(x) && aligned16(g) && aligned16(b) && aligned16(y);
  int64_t packs = cols / N;
  if (vec && packs <= 32 * 16) {
    // persistent: up to four CTAs of eight warps per SM, every warp walks rows with two in flight
    const int threads = 256, wpb = 8;
    // CTAs per SM (APPLEGPU_LN_BPS overrides): measured best on [8192, 768] at 2 for 16-bit rows and 4 for float32
    static const int bps_env = [] { const char* v = std::getenv("APPLEGPU_LN_BPS"); int n = v ? std::atoi(v) : 0; return n < 0 ? 0 : n > 8 ? 8 : n; }();
    const int bps = bps_env ? bps_env : (sizeof(T) == 4 ? 4 : 2);
    int grid = grid_for(rows, wpb, bps);
    int iters = (int)((packs + 31) / 32);
    cudaError_t le = cudaSuccess;
    if constexpr (sizeof(T) == 2) {
      int* status = matmul_status_word();
      const int from = iters >= 5 ? 32 : iters == 4 ? (std::is_same<T, __half>::value ? 160 : 32) : iters == 2 ? 64 : 112;      // rows an SM
      if (status && cols * 2 >= kSmMinRowBytes && cols * 2 <= kLnMaxRowBytes && rows >= from * (int64_t)sm_count() && x != y) {
#define AG_LNB(I) le = launch_layer_norm_bulk<T, I>(s, x, g, b, y, rows, (int)cols, eps, status)
        if (iters <= 2) AG_LNB(2); else if (iters <= 3) AG_LNB(3); else if (iters <= 4) AG_LNB(4); else AG_LNB(5);
#undef AG_LNB
        return cuda_status(le, "layer_norm");
      }
    }
#define AG_LN(I) le = launch_pdl(layer_norm_warp_kernel<T, I>, dim3(grid), dim3(threads), 0, s, x, g, b, y, rows, (int)cols, eps)
    if (iters <= 1) AG_LN(1); else if (iters <= 2) AG_LN(2); else if (iters <= 3) AG_LN(3); else if (iters <= 4) AG_LN(4);
    else if (iters <= 6) AG_LN(6); else if (iters <= 8) AG_LN(8); else if (iters <= 12) AG_LN(12); else AG_LN(16);
#undef AG_LN
    if (le != cudaSuccess) return cuda_status(le, "layer_norm");
  } else {
    int grid = (int)(rows < (int64_t)sm_count() * 8 ? rows : (int64_t)sm_count() * 8);
    layer_norm_block_kernel<T><<<grid, 256, 0, s>>>(x, g, b, y, rows, cols, eps);
  }
  AG_CHECK_LAUNCH("layer_norm");
  return Status::OK();
}

Status layer_norm(cudaStream_t s, const TView& in, const TView& gamma, const TView& beta, float eps, const TView& out) {
  if (!in.contiguous() || !out.contiguous() || !gamma.contiguous() || !beta.contiguous())
    return Status::compute("layer_norm needs contiguous tensors");
  if (gamma.dtype != in.dtype || beta.dtype != in.dtype) return Status::invalid("layer_norm gamma/beta dtype must match input");
  AG_DISPATCH_FLOAT(in.dtype, T, return layer_norm_t<T>(s, in, gamma, beta, eps, out));
  return Status::OK();
}

// ── softmax / softmax_causal ────────────────────────────────────────────────
// One row in a warp's registers: `valid` unmasked leading columns; put(pack index, results) for every pack of the row.
// 16-bit rows stay as words of two, and arithmetic is on pairs: a row of 1024 took 509 instructions element by element (63 % of the
// issue slots at 40 % of the memory's rate) and takes about half of them now. The exponential is 2^24 exp(x - max) for bfloat16, the factor
// leaving with the sum: the hardware's exp2 gives zero for what it would not hold as a normal number, and this way that is nothing bfloat16 holds.
template <typename T, int ITERS, bool CAUSAL, typename Put>
__device__ __forceinline__ void softmax_row16(const Pack<T> (&cur)[ITERS], int lane, int packs, int valid, Put put) {
  constexpr uint32_t kNegInf = std::is_same<T, __half>::value ? 0xfc00u : 0xff80u;
  uint4 x[ITERS];
  uint32_t top = kNegInf | kNegInf << 16;
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    const int pk = lane + it * 32, left = valid - pk * 8;
    if (pk >= packs || left <= 0) continue;
    x[it] = reinterpret_cast<const uint4&>(cur[it]);
    if (left < 8) {                                        // the pack the diagonal crosses
      uint32_t* w = reinterpret_cast<uint32_t*>(&x[it]);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (2 * j >= left) w[j] = kNegInf | kNegInf << 16;
        else if (2 * j + 1 >= left) w[j] = (w[j] & 0xffffu) | kNegInf << 16;
      }
    }
    top = max_word<T>(max_word<T>(top, max_word<T>(x[it].x, x[it].y)), max_word<T>(x[it].z, x[it].w));
  }
  float lo, hi;
  unpack_f32x2(widen_word<T>(top), lo, hi);
  const float m = warp_max(fmaxf(fmaxf(lo, hi), CAUSAL ? -1e9f : -INFINITY));
  constexpr float kLog2e = 1.4426950408889634f, kUp = std::is_same<T, __half>::value ? 0.f : 24.f;
  const uint64_t nm = pack_f32x2(-m, -m), scale = pack_f32x2(kLog2e, kLog2e), up = pack_f32x2(kUp, kUp);
  uint64_t sums = 0;                                       // the bits of (0.f, 0.f)
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    const int pk = lane + it * 32;
    if (pk >= packs || pk * 8 >= valid) continue;
    uint32_t* w = reinterpret_cast<uint32_t*>(&x[it]);
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float a, b;
      unpack_f32x2(fma_f32x2(add_f32x2(widen_word<T>(w[j]), nm), scale, up), a, b);
      a = ex2_approx(a); b = ex2_approx(b);
      sums = add_f32x2(sums, pack_f32x2(a, b));
      w[j] = pack2_t<T>(a, b);                             // the reference stores exp() in the storage type and divides that value
    }
  }
  const float inv = __fdiv_rn(1.0f, warp_sum(sum_f32x2(sums)));      // one division per row; e * (1/sum) is within 1 ulp of e / sum
  const uint64_t inv2 = pack_f32x2(inv, inv);
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    const int pk = lane + it * 32;
    if (pk >= packs) continue;
    uint4 o = make_uint4(0u, 0u, 0u, 0u);
    if (pk * 8 < valid) {
      uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float a, b;
        unpack_f32x2(mul_f32x2(widen_word<T>(reinterpret_cast<const uint32_t*>(&x[it])[j]), inv2), a, b);
        w[j] = pack2_t<T>(a, b);
      }
    }
    put(pk, reinterpret_cast<const Pack<T>&>(o));
  }
}
template <typename T, int ITERS, bool CAUSAL, bool WORDS, typename Put>
__device__ __forceinline__ void softmax_row(const Pack<T> (&cur)[ITERS], int lane, int packs, int valid, Put put) {
  if constexpr (WORDS) { softmax_row16<T, ITERS, CAUSAL>(cur, lane, packs, valid, put); return; }
  constexpr int N = Pack<T>::N;
  float v[ITERS][N];
  float m = CAUSAL ? -1e9f : -INFINITY;
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    const int c0 = (lane + it * 32) * N;
    if (lane + it * 32 < packs && c0 < valid) {
      if (c0 + N <= valid) {
#pragma unroll
        for (int e = 0; e < N; e++) { v[it][e] = Cvt<T>::to(cur[it].v[e]); m = fmaxf(m, v[it][e]); }
      } else {
#pragma unroll
        for (int e = 0; e < N; e++) {
          const float f = Cvt<T>::to(cur[it].v[e]);
          const bool on = c0 + e < valid;
          v[it][e] = on ? f : -INFINITY;
          if (on) m = fmaxf(m, f);
        }
      }
    }
  }
  m = warp_max(m);
  float sum = 0.f;
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    // packs entirely right of the diagonal (or past the row) hold only masked slots: skip their math
    if ((lane + it * 32) * N < valid && lane + it * 32 < packs) {
#pragma unroll
      for (int e = 0; e < N; e++) {
        // Masked slots hold -inf and contribute exp(-inf) = 0. __expf (hardware exp2) is within
        // 2 ulp plus the rounding of x*log2(e): well inside the 1e-5 bar.
        float ex = __expf(v[it][e] - m);
        sum += ex;
        // Half types: the reference stores exp() in the storage type and divides that value.
        v[it][e] = Cvt<T>::to(Cvt<T>::from(ex));
      }
    }
  }
  sum = warp_sum(sum);
  const float inv = __fdiv_rn(1.0f, sum);  // one division per row; e * (1/sum) is within 1 ulp of e / sum
#pragma unroll
  for (int it = 0; it < ITERS; it++) {
    int pk = lane + it * 32;
    int c0 = pk * N;
    if (pk < packs) {
      Pack<T> o;
      if (c0 < valid) {
        float r[N];
#pragma unroll
        for (int e = 0; e < N; e++) r[e] = v[it][e] * inv;     // masked slots hold exp(-inf) = 0: they store 0
        pack_from_floats<T>(o, r);
      } else {
#pragma unroll
        for (int e = 0; e < N; e++) o.v[e] = Cvt<T>::from(0.f);
      }
      put(pk, o);
    }
  }
}
template <bool CAUSAL>
__device__ __forceinline__ int softmax_valid(int64_t row, int64_t total_rows, int rows_per_mat, int cols) {
  if (!CAUSAL) return cols;
  // 32-bit remainder where the row count allows it: the 64-bit one costs about a fifth of a 1024-column row
  const int r = total_rows <= 0x7fffffff ? (int)((unsigned int)row % (unsigned int)rows_per_mat) : (int)(row % rows_per_mat);
  return r + 1 < cols ? r + 1 : cols;
}
// Warp-per-row with the row in registers; `valid` = number of unmasked leading columns. A persistent grid walks the
// rows and a warp keeps two rows in flight: the 16-byte loads of its next row are issued before the reductions of the
// current one (a row's chain load -> max -> exp -> sum -> store is latency-bound on its own). Packs wholly left of the
// diagonal take a mask-free path, the one pack the diagonal crosses is masked per element, packs right of it are
// neither read nor computed: zeros are stored.
// Rows of one pack a lane are too short for the word form, which has the longer chain: 1850 x 128 x 128 bfloat16 69.7 us element by element, 96.4 by
// words, float16 64.6 / 97.2, causal 84.4 / 117.1; only causal bfloat16 gains, 124.3 / 117.0.
template <typename T, int ITERS, bool CAUSAL> constexpr bool softmax_words = sizeof(T) == 2 && (ITERS > 1 || (CAUSAL && std::is_same<T, __nv_bfloat16>::value));
template <typename T, int ITERS, bool CAUSAL>
__global__ void __launch_bounds__(128, 4) softmax_warp_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t total_rows, int rows_per_mat, int cols) {
  constexpr int N = Pack<T>::N;
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const int packs = cols / N;
  pdl_wait();
  pdl_trigger();
  auto valid_of = [&](int64_t row) { return softmax_valid<CAUSAL>(row, total_rows, rows_per_mat, cols); };
  const int64_t stride = (int64_t)gridDim.x * wpb;
  int64_t row = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5);
  Pack<T> cur[ITERS], nxt[ITERS];
  int valid = 0;
  if (row < total_rows) {
    valid = valid_of(row);
#pragma unroll
    for (int it = 0; it < ITERS; it++) { int pk = lane + it * 32; if (pk < packs && pk * N < valid) cur[it] = ld16_stream(in + row * cols + pk * N); }
  }
  for (; row < total_rows; row += stride) {
    const int64_t next = row + stride;
    int next_valid = 0;
    if (next < total_rows) {
      next_valid = valid_of(next);
#pragma unroll
      for (int it = 0; it < ITERS; it++) { int pk = lane + it * 32; if (pk < packs && pk * N < next_valid) nxt[it] = ld16_stream(in + next * cols + pk * N); }
    }
    T* y = out + row * cols;
    softmax_row<T, ITERS, CAUSAL, softmax_words<T, ITERS, CAUSAL>>(cur, lane, packs, valid, [&](int pk, const Pack<T>& o) { st16_stream(y + pk * N, o); });
#pragma unroll
    for (int it = 0; it < ITERS; it++) cur[it] = nxt[it];
    valid = next_valid;
  }
}

// The same with rows that come and go by bulk copies. A warp has kSmSlots row buffers in shared memory: one lane asks for a row's
// unmasked part three rows ahead, the row is computed in place, and the whole row leaves as one copy, zeros included. No register holds a row
// that is on its way, so more warps fit an SM.
// For rows of 512 to 2048 bytes (4096 of float32), from 32 of them an SM on (the warps of the form above ask for their third row there), of less than
// 768 bytes from 80. Rows in registers against bulk copies, causal, us: bfloat16 96 x
// 1024 x 1024 65.4 / 59.6, 96 x 512 x 512 34.4 / 23.6, 96 x 256 x 256 14.5 / 10.8, 96 x 128 x 128 6.3 / 6.8, 3 x 1024 x 1024 4.9 /
// 5.5, 8 x 2048 x 2048 20.5 / 25.5; float32 112.9 / 106.4, 36.6 / 27.7, 15.8 / 11.5, 6.8 / 6.1, 6.6 / 6.7, 61 / 82; rows of 512 bytes at 32, 64 and 97
// an SM, float32 3.6 / 4.1, 5.0 / 5.2, 7.7 / 6.4, 256 of bfloat16 3.7 / 3.9, 5.3 / 5.7, 9.1 / 7.1. (Element by element,
// in registers, the first took 72: it was bound by instructions.) What bounds it now: memory, 302 MB at 5.1 TB/s.
// Without a mask: bfloat16 48 x 1024 x 1024 42.8 / 36.1, 382 x 256 x 256 43.8 / 27.6; float32 382 x 256 x 256 51.1 / 37.8, 64 x 768 x 768 57.7 / 55.2.
// float32 rows of more than 2048 bytes and 160 MB in all stay in registers, whose loads and stores do not push one another out of the L2: 127 x
// 768 x 768 110.0 / 110.8, 254 215 / 221, 48 x 1024 x 1024 68.4 / 73.6, 191 255 / 290; 64 x 768 x 768 (151 MB) and less as above.
template <typename T> constexpr int kSmMaxRowBytes = sizeof(T) == 4 ? 4096 : 2048;
template <typename T, int ITERS, bool CAUSAL>
__global__ void __launch_bounds__(kSmWarps * 32) softmax_bulk_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t total_rows, int rows_per_mat, int cols, int* status) {
  constexpr int N = Pack<T>::N;
  extern __shared__ __align__(128) uint8_t s_rows[];
  __shared__ uint64_t bars[kSmWarps][kSmSlots];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int packs = cols / N, row_bytes = cols * (int)sizeof(T);
  uint8_t* const mine = s_rows + (size_t)warp * kSmSlots * row_bytes;
  uint64_t* const bar = bars[warp];
  if (lane == 0) {
    for (int i = 0; i < kSmSlots; i++) sm100::mbar_init(&bar[i], 1);
    sm100::mbar_fence_init();
  }
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  const int64_t stride = (int64_t)gridDim.x * kSmWarps, row0 = (int64_t)blockIdx.x * kSmWarps + warp;
  auto ask = [&](int64_t row, int slot) {                    // one lane
    bulk_load(mine + slot * row_bytes, in + row * cols, (uint32_t)((softmax_valid<CAUSAL>(row, total_rows, rows_per_mat, cols) + N - 1) / N * 16), &bar[slot]);
  };
  int64_t asked = row0;                                      // the next row to ask for
  if (lane == 0) {
    for (int i = 0; i < kSmSlots - 1 && asked < total_rows; i++, asked += stride) ask(asked, i);
  }
  int slot = 0, free_slot = kSmSlots - 1;
  uint32_t phase = 0;
  int64_t row = row0;
  for (; row < total_rows; row += stride) {
    if (lane == 0 && asked < total_rows) {
      // the free slot held the row just done: its copy out must have read it (a warp waits here, the SM has others)
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      ask(asked, free_slot);
      asked += stride;
    }
    if (!__all_sync(0xffffffffu, sm100::mbar_wait_limit(&bar[slot], phase, status, 9))) break;
    const int valid = softmax_valid<CAUSAL>(row, total_rows, rows_per_mat, cols);
    uint4* const at = reinterpret_cast<uint4*>(mine + slot * row_bytes);
    Pack<T> cur[ITERS];
#pragma unroll
    for (int it = 0; it < ITERS; it++) {
      const int pk = lane + it * 32;
      if (pk < packs && pk * N < valid) *reinterpret_cast<uint4*>(&cur[it]) = at[pk];
    }
    softmax_row<T, ITERS, CAUSAL, sizeof(T) == 2>(cur, lane, packs, valid, [&](int pk, const Pack<T>& o) { at[pk] = *reinterpret_cast<const uint4*>(&o); });
    sm100::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) bulk_store(out + row * cols, at, (uint32_t)row_bytes);
    free_slot = slot;
    if (++slot == kSmSlots) { slot = 0; phase ^= 1; }
  }
  if (lane == 0) bulk_leave(bar, row, asked, stride, slot, phase, status);
}
template <typename T, int ITERS, bool CAUSAL>
static cudaError_t launch_softmax_bulk(cudaStream_t s, const T* x, T* y, int64_t total_rows, int64_t rows_per_mat, int64_t cols, int* status) {
  const int smem = kSmWarps * kSmSlots * (int)(cols * (int64_t)sizeof(T));
  auto kern = softmax_bulk_kernel<T, ITERS, CAUSAL>;
  static int by_registers = 0;
  int per_sm;
  cudaError_t e = bulk_ctas(kern, smem, kSmMaxRowBytes<T>, &by_registers, &per_sm);
  if (e != cudaSuccess) return e;
  return launch_pdl(kern, dim3((unsigned)grid_for(total_rows, kSmWarps, per_sm)), dim3(kSmWarps * 32), (size_t)smem, s, x, y, total_rows, (int)rows_per_mat, (int)cols, status);
}

// Block-per-row for long or unaligned rows.
template <typename T, bool CAUSAL>
__global__ void __launch_bounds__(256) softmax_block_kernel(const T* in, T* out, int64_t total_rows, int64_t rows_per_mat, int64_t cols) {
  __shared__ float red[33];
  for (int64_t row = blockIdx.x; row < total_rows; row += gridDim.x) {
    int64_t valid = cols;
    if (CAUSAL) { int64_t r = row % rows_per_mat; valid = r + 1 < cols ? r + 1 : cols; }
    const T* x = in + row * cols;
    float m = CAUSAL ? -1e9f : -INFINITY;
    for (int64_t j = threadIdx.x; j < valid; j += blockDim.x) m = fmaxf(m, Cvt<T>::to(x[j]));
    m = block_max(m, red);
    float sum = 0.f;
    for (int64_t j = threadIdx.x; j < valid; j += blockDim.x) sum += expf(Cvt<T>::to(x[j]) - m);
    sum = block_sum(sum, red);
    T* y = out + row * cols;
    for (int64_t j = threadIdx.x; j < cols; j += blockDim.x) {
      if (j < valid) {
        float e = Cvt<T>::to(Cvt<T>::from(expf(Cvt<T>::to(x[j]) - m)));
        y[j] = Cvt<T>::from(__fdiv_rn(e, sum));
      } else y[j] = Cvt<T>::from(0.f);
    }
  }
}

template <typename T, bool CAUSAL>
static Status softmax_t(cudaStream_t s, const TView& in, const TView& out) {
  constexpr int N = Pack<T>::N;
  int64_t cols = in.shape.back();
  if (cols == 0 || in.numel() == 0) return Status::OK();
  int64_t total_rows = in.numel() / cols;
  int64_t rows_per_mat = CAUSAL ? in.shape[in.nd() - 2] : 1;
  const T* x = (const T*)in.ptr; T* y = (T*)out.ptr;
  int64_t packs = cols / N;
  bool vec = cols % N == 0 && aligned16(x) && aligned16(y) && packs <= 32 * 16 && in.ptr != out.ptr;
  if (vec) {
    // persistent: four CTAs of four warps per SM (the kernel keeps two rows per warp in registers: ~128 registers)
    const int threads = 128, wpb = 4;
    int grid = grid_for(total_rows, wpb, 4);
    int iters = (int)((packs + 31) / 32);
    cudaError_t le = cudaSuccess;
    int* status = matmul_status_word();
    const int64_t row_bytes = cols * (int64_t)sizeof(T);
    const bool large = !CAUSAL && row_bytes > 2048 && total_rows * row_bytes > (160ll << 20);      // float32
    if (status && row_bytes >= kSmMinRowBytes && row_bytes <= kSmMaxRowBytes<T> && total_rows >= (row_bytes < 768 ? 80 : 32) * (int64_t)sm_count() && !large) {
#define AG_SMB(I) le = launch_softmax_bulk<T, I, CAUSAL>(s, x, y, total_rows, rows_per_mat, cols, status)
      if (iters <= 1) AG_SMB(1); else if (iters <= 2) AG_SMB(2); else if (iters <= 4) AG_SMB(4); else AG_SMB(8);
#undef AG_SMB
    } else
#define AG_SM(I) le = launch_pdl(softmax_warp_kernel<T, I, CAUSAL>, dim3(grid), dim3(threads), 0, s, x, y, total_rows, (int)rows_per_mat, (int)cols)
    if (iters <= 1) AG_SM(1); else if (iters <= 2) AG_SM(2); else if (iters <= 4) AG_SM(4);
    else if (iters <= 8) AG_SM(8); else AG_SM(16);
#undef AG_SM
    if (le != cudaSuccess) return cuda_status(le, "softmax");
  } else {
    int grid = (int)(total_rows < (int64_t)sm_count() * 8 ? total_rows : (int64_t)sm_count() * 8);
    softmax_block_kernel<T, CAUSAL><<<grid, 256, 0, s>>>(x, y, total_rows, rows_per_mat, cols);
  }
  AG_CHECK_LAUNCH("softmax");
  return Status::OK();
}

Status softmax(cudaStream_t s, const TView& in, bool causal, const TView& out) {
  if (!in.contiguous() || !out.contiguous()) return Status::compute("softmax needs contiguous tensors");
  if (causal) { AG_DISPATCH_FLOAT(in.dtype, T, return (softmax_t<T, true>(s, in, out))); }
  else { AG_DISPATCH_FLOAT(in.dtype, T, return (softmax_t<T, false>(s, in, out))); }
  return Status::OK();
}

// ── argmax ──────────────────────────────────────────────────────────────────
// Serial-scan semantics: result = lowest index holding the maximum over non-NaN elements,
// except that a NaN in element 0 is never displaced (every '>' against NaN is false).
struct ArgPair { float v; int i; };
__device__ __forceinline__ ArgPair arg_better(ArgPair a, ArgPair b) {
  // a and b are both "valid" candidates (i >= 0); invalid carries i = INT_MAX and v = -inf.
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
// One block per row, whose time is its rounds of loads: long rows that leave SMs idle take blocks of 1024 threads (eight rows of 32768
// floats in a step: 18.50 -> 18.34 ms for 49 steps, about 3 us a launch).
template <typename T>
__global__ void __launch_bounds__(1024) argmax_kernel(const T* __restrict__ in, int32_t* __restrict__ out, int64_t rows, int64_t cols, int64_t row_stride) {
  __shared__ float sv[32];
  __shared__ int si[32];
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const T* x = in + row * row_stride;
    ArgPair best{-INFINITY, 0x7fffffff};
    // Each thread visits its elements in ascending index order, so a strict '>' keeps the first
    // maximum; NaNs never compare greater. Rows start on arbitrary element boundaries (a 50257-wide
    // row is only 2-byte aligned): scalar head up to the first 16-byte boundary, 16-byte packs, scalar tail.
    constexpr int N = Pack<T>::N;
    int64_t head = (int64_t)(((16u - (unsigned)(reinterpret_cast<uintptr_t>(x) & 15u)) & 15u) / sizeof(T));
    if (head > cols) head = cols;
    for (int64_t j = threadIdx.x; j < head; j += blockDim.x) {
      float f = Cvt<T>::to(x[j]);
      if (f > best.v) best = ArgPair{f, (int)j};
    }
    const int64_t npacks = (cols - head) / N;
    const T* xv = x + head;
    int64_t pk = threadIdx.x;
    for (; pk + 3 * (int64_t)blockDim.x < npacks; pk += 4 * (int64_t)blockDim.x) {
      Pack<T> q[4];
#pragma unroll
      for (int u = 0; u < 4; u++) q[u] = ld16_stream(xv + (pk + u * (int64_t)blockDim.x) * N);
#pragma unroll
      for (int u = 0; u < 4; u++) {
#pragma unroll
        for (int e = 0; e < N; e++) {
          float f = Cvt<T>::to(q[u].v[e]);
          if (f > best.v) best = ArgPair{f, (int)(head + (pk + u * (int64_t)blockDim.x) * N + e)};
        }
      }
    }
    for (; pk < npacks; pk += blockDim.x) {
      Pack<T> q = ld16_stream(xv + pk * N);
#pragma unroll
      for (int e = 0; e < N; e++) {
        float f = Cvt<T>::to(q.v[e]);
        if (f > best.v) best = ArgPair{f, (int)(head + pk * N + e)};
      }
    }
    for (int64_t j = head + npacks * N + threadIdx.x; j < cols; j += blockDim.x) {
      float f = Cvt<T>::to(x[j]);
      if (f > best.v) best = ArgPair{f, (int)j};
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgPair other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = arg_better(best, other);
    }
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) { sv[w] = best.v; si[w] = best.i; }
    __syncthreads();
    if (w == 0) {
      ArgPair b2 = lane < nw ? ArgPair{sv[lane], si[lane]} : ArgPair{-INFINITY, 0x7fffffff};
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ArgPair other{__shfl_xor_sync(0xffffffffu, b2.v, o), __shfl_xor_sync(0xffffffffu, b2.i, o)};
        b2 = arg_better(b2, other);
      }
      if (lane == 0) {
        float x0 = Cvt<T>::to(x[0]);
        int r = b2.i;
        if (x0 != x0 || r == 0x7fffffff) r = 0;  // NaN at 0 sticks; all-NaN row -> 0
        out[row] = r;
      }
    }
  }
}
// Integer rows (the reference allows every dtype but Bool): compare natively.
template <typename T>
__global__ void argmax_int_kernel(const T* __restrict__ in, int32_t* __restrict__ out, int64_t rows, int64_t cols) {
  int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (row >= rows) return;
  const T* x = in + row * cols;
  T best = x[0]; int idx = 0;
  for (int64_t j = 1; j < cols; j++) if (x[j] > best) { best = x[j]; idx = (int)j; }
  out[row] = idx;
}

Status argmax(cudaStream_t s, const TView& in, const TView& out) {
  // rows dense, or all at one pitch (last stride 1, leading dims collapsing onto the row stride)
  int64_t cols = in.shape.back();
  if (cols == 0) return Status::compute("argmax over an empty row");
  int64_t rows = in.numel() / cols;
  int64_t row_stride = cols;
  if (!in.contiguous()) {
    if (in.shape.size() < 2 || in.strides.back() != 1) return Status::compute("argmax needs dense rows");
    row_stride = in.strides[in.shape.size() - 2];
    if (in.dtype != DType::F32 && in.dtype != DType::F16 && in.dtype != DType::BF16) return Status::compute("argmax needs a contiguous tensor");
  }
  if (rows == 0) return Status::OK();
  int grid = (int)(rows < (int64_t)sm_count() * 8 ? rows : (int64_t)sm_count() * 8);
  const int threads = rows <= sm_count() && cols >= 8192 ? 1024 : 256;
  switch (in.dtype) {
    case DType::F32: argmax_kernel<float><<<grid, threads, 0, s>>>((const float*)in.ptr, (int32_t*)out.ptr, rows, cols, row_stride); break;
    case DType::F16: argmax_kernel<__half><<<grid, threads, 0, s>>>((const __half*)in.ptr, (int32_t*)out.ptr, rows, cols, row_stride); break;
    case DType::BF16: argmax_kernel<__nv_bfloat16><<<grid, threads, 0, s>>>((const __nv_bfloat16*)in.ptr, (int32_t*)out.ptr, rows, cols, row_stride); break;
    case DType::I32: argmax_int_kernel<int32_t><<<(int)((rows + 127) / 128), 128, 0, s>>>((const int32_t*)in.ptr, (int32_t*)out.ptr, rows, cols); break;
    case DType::I64: argmax_int_kernel<int64_t><<<(int)((rows + 127) / 128), 128, 0, s>>>((const int64_t*)in.ptr, (int32_t*)out.ptr, rows, cols); break;
    case DType::U8: argmax_int_kernel<uint8_t><<<(int)((rows + 127) / 128), 128, 0, s>>>((const uint8_t*)in.ptr, (int32_t*)out.ptr, rows, cols); break;
    case DType::U32: argmax_int_kernel<uint32_t><<<(int)((rows + 127) / 128), 128, 0, s>>>((const uint32_t*)in.ptr, (int32_t*)out.ptr, rows, cols); break;
    case DType::I8: argmax_int_kernel<int8_t><<<(int)((rows + 127) / 128), 128, 0, s>>>((const int8_t*)in.ptr, (int32_t*)out.ptr, rows, cols); break;
    case DType::I16: argmax_int_kernel<int16_t><<<(int)((rows + 127) / 128), 128, 0, s>>>((const int16_t*)in.ptr, (int32_t*)out.ptr, rows, cols); break;
    default: return Status::unsupported("Argmax does not support bool dtype");
  }
  AG_CHECK_LAUNCH("argmax");
  return Status::OK();
}

// ── sums ────────────────────────────────────────────────────────────────────
// out[o, i] = sum_r in[o, r, i]   (outer, reduce, inner) — serves sum_dim and sum over last dim.
template <typename T>
__global__ void __launch_bounds__(256) sum_mid_kernel(const T* __restrict__ in, T* __restrict__ out, int64_t outer, int64_t red, int64_t inner, float scale) {
  if (inner == 1) {
    __shared__ float sm[33];
    for (int64_t o = blockIdx.x; o < outer; o += gridDim.x) {
      float s = 0.f;
      for (int64_t r = threadIdx.x; r < red; r += blockDim.x) s += Cvt<T>::to(in[o * red + r]);
      s = block_sum(s, sm);
      if (threadIdx.x == 0) out[o] = Cvt<T>::from(s * scale);
    }
  } else {
    int64_t n = outer * inner;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
      int64_t o = i / inner, c = i % inner;
      float s = 0.f;
      for (int64_t r = 0; r < red; r++) s += Cvt<T>::to(in[(o * red + r) * inner + c]);
      out[i] = Cvt<T>::from(s * scale);
    }
  }
}
static Status sum_mid(cudaStream_t s, const TView& in, const TView& out, int64_t outer, int64_t red, int64_t inner, float scale) {
  if (!in.contiguous()) return Status::compute("sum needs a contiguous tensor");
  if (outer * inner == 0) return Status::OK();
  int grid = inner == 1 ? (int)(outer < (int64_t)sm_count() * 8 ? outer : (int64_t)sm_count() * 8) : grid_for(outer * inner, 256, 8);
  AG_DISPATCH_FLOAT(in.dtype, T, (sum_mid_kernel<T><<<grid, 256, 0, s>>>((const T*)in.ptr, (T*)out.ptr, outer, red, inner, scale)));
  AG_CHECK_LAUNCH("sum");
  return Status::OK();
}
Status sum_last(cudaStream_t s, const TView& in, const TView& out, bool mean) {
  int64_t cols = in.shape.empty() ? 1 : in.shape.back();
  int64_t rows = cols ? in.numel() / cols : 0;
  return sum_mid(s, in, out, rows, cols, 1, mean && cols ? 1.0f / (float)cols : 1.0f);
}
Status sum_dim(cudaStream_t s, const TView& in, int dim, const TView& out) {
  int64_t outer = 1, inner = 1;
  for (int d = 0; d < dim; d++) outer *= in.shape[d];
  for (int d = dim + 1; d < in.nd(); d++) inner *= in.shape[d];
  return sum_mid(s, in, out, outer, in.shape[dim], inner, 1.0f);
}
Status mean_all(cudaStream_t s, const TView& in, const TView& out) {
  int64_t n = in.numel();
  return sum_mid(s, in, out, 1, n, 1, n ? 1.0f / (float)n : 1.0f);
}

}}  // namespace ag::k
