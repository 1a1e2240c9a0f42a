// Attention of heads that share keys and values in groups, over a cache of normed, turned keys and plain values.
//
//   append  a warp per head and row: RMS norm over the head, the rotation of its first entries (i with i + rot_pairs), queries in
//           place, keys and values into the cache
//   decode  short portions: a cluster per (row, key head), each CTA a split of the keys the row sees, for up to eight query heads
//           at a time; the splits meet over distributed shared memory. Scores, their maximum and the weights are float32.
// Longer portions take prompt_attention straight over the cache.
#include "common.cuh"
#include "seq_kernels.h"
#include "sm100.cuh"
#include <algorithm>

namespace ag { namespace k {

struct GaParams {
  void* proj; const float* q_norm; const float* k_norm; const float2* rot; void* cache; const int* pos; void* y;
  long long ld, seq_stride, y_ld, cld, v_col;
  int n_seq, T, heads, kv_heads, group, dim, vdim, pairs, window, shared, max_len, q_off, k_off, v_off;
  int hg, h_parts;                       // query heads per CTA, CTAs along a group's heads
  int paired;                            // append: every column turns, a lane takes two neighbours of either half at a time
  float scale, cap, eps;
};

static Status ga_params(const GroupedAttnDesc& d, GaParams* out) {
  if (d.n_seq < 1 || d.T < 1 || d.heads < 1 || d.kv_heads < 1 || d.heads % d.kv_heads || d.dim < 1 || d.vdim < 1 || d.rot_pairs < 0 || 2 * d.rot_pairs > d.dim || d.window < 0)
    return Status::invalid("grouped attention: bad sizes");
  if (!d.proj || !d.cache || !d.pos || !d.q_norm || (!d.shared && !d.k_norm) || (d.rot_pairs && !d.rot_table)) return Status::invalid("grouped attention: missing operand");
  GaParams& p = *out;
  p.proj = d.proj; p.q_norm = d.q_norm; p.k_norm = d.k_norm; p.rot = d.rot_table; p.cache = d.cache; p.pos = d.pos; p.y = d.y;
  p.ld = d.ld; p.seq_stride = d.seq_stride; p.y_ld = d.y_ld; p.cld = grouped_cache_ld(d.kv_heads, d.dim, d.vdim); p.v_col = grouped_v_col(d.kv_heads, d.dim);
  p.n_seq = d.n_seq; p.T = d.T; p.heads = d.heads; p.kv_heads = d.kv_heads; p.group = d.heads / d.kv_heads; p.dim = d.dim; p.vdim = d.vdim; p.pairs = d.rot_pairs;
  p.window = d.window; p.shared = d.shared ? 1 : 0; p.max_len = d.max_len; p.q_off = d.q_off; p.k_off = d.k_off; p.v_off = d.v_off;
  p.scale = d.scale; p.cap = d.softcap; p.eps = d.eps; p.hg = 1; p.h_parts = 1; p.paired = 0;
  return Status::OK();
}

// ── append ──────────────────────────────────────────────────────────────────
constexpr int kGaThreads = 256;
template <typename T>
__device__ __forceinline__ void ga_norm_turn(const GaParams& p, const T* src, T* dst, const float* w, int position, int lane) {
  float sq = 0.f;
  for (int i = lane; i < p.dim; i += 32) { const float v = Cvt<T>::to(src[i]); sq = fmaf(v, v, sq); }
  const float rs = 1.0f / sqrtf(warp_sum(sq) / (float)p.dim + p.eps);       // also: every lane has read before any writes
  for (int i = lane; i < p.pairs; i += 32) {
    const float2 cs = p.rot[(long long)position * p.pairs + i];
    const float u = Cvt<T>::to(src[i]) * rs * w[i], v = Cvt<T>::to(src[i + p.pairs]) * rs * w[i + p.pairs];
    dst[i] = Cvt<T>::from(u * cs.x - v * cs.y);
    dst[i + p.pairs] = Cvt<T>::from(v * cs.x + u * cs.y);
  }
  for (int i = 2 * p.pairs + lane; i < p.dim; i += 32) dst[i] = Cvt<T>::from(Cvt<T>::to(src[i]) * rs * w[i]);
}
// The same for 16-bit heads that turn as a whole (dim = 2 pairs <= 256, everything on the accesses' alignment): two neighbouring columns of
// either half at a time, all of a lane's operands asked for at once and read once.
template <typename T>
__device__ __forceinline__ void ga_norm_turn_pairs(const GaParams& p, const T* src, T* dst, const float* w, int position, int lane) {
  constexpr int IT = 2;                  // pairs <= 128
  uint32_t a[IT], b[IT];
  float2 wa[IT], wb[IT];
  float4 cs[IT];
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = 2 * lane + 64 * it;
    a[it] = b[it] = 0u; wa[it] = wb[it] = make_float2(0.f, 0.f); cs[it] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i >= p.pairs) continue;
    a[it] = *reinterpret_cast<const uint32_t*>(src + i); b[it] = *reinterpret_cast<const uint32_t*>(src + i + p.pairs);
    wa[it] = *reinterpret_cast<const float2*>(w + i); wb[it] = *reinterpret_cast<const float2*>(w + i + p.pairs);
    cs[it] = *reinterpret_cast<const float4*>(p.rot + (long long)position * p.pairs + i);
  }
  auto wide = [](uint32_t v) {
    const T* e = reinterpret_cast<const T*>(&v);
    return make_float2(Cvt<T>::to(e[0]), Cvt<T>::to(e[1]));
  };
  float sq = 0.f;
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const float2 u = wide(a[it]), v = wide(b[it]);
    sq = fmaf(u.x, u.x, fmaf(u.y, u.y, fmaf(v.x, v.x, fmaf(v.y, v.y, sq))));
  }
  const float rs = 1.0f / sqrtf(warp_sum(sq) / (float)p.dim + p.eps);
#pragma unroll
  for (int it = 0; it < IT; it++) {
    const int i = 2 * lane + 64 * it;
    if (i >= p.pairs) continue;
    float2 u = wide(a[it]), v = wide(b[it]);
    u.x *= rs * wa[it].x; u.y *= rs * wa[it].y; v.x *= rs * wb[it].x; v.y *= rs * wb[it].y;
    alignas(4) T lo[2] = {Cvt<T>::from(u.x * cs[it].x - v.x * cs[it].y), Cvt<T>::from(u.y * cs[it].z - v.y * cs[it].w)};
    alignas(4) T hi[2] = {Cvt<T>::from(v.x * cs[it].x + u.x * cs[it].y), Cvt<T>::from(v.y * cs[it].z + u.y * cs[it].w)};
    *reinterpret_cast<uint32_t*>(dst + i) = *reinterpret_cast<const uint32_t*>(lo);
    *reinterpret_cast<uint32_t*>(dst + i + p.pairs) = *reinterpret_cast<const uint32_t*>(hi);
  }
}
template <typename T, bool PAIRED>
__global__ void __launch_bounds__(kGaThreads) grouped_append_kernel(const GaParams p) {
  auto norm_turn = [&](const T* src, T* dst, const float* w, int position, int lane) {
    if constexpr (PAIRED) ga_norm_turn_pairs<T>(p, src, dst, w, position, lane); else ga_norm_turn<T>(p, src, dst, w, position, lane);
  };
  pdl_wait();
  pdl_trigger();
  const int r = blockIdx.x, s = r / p.T, t = r % p.T, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int position = p.pos[s] + t;
  if (position < 0 || position >= p.max_len) return;
  T* row = reinterpret_cast<T*>(p.proj) + (long long)r * p.ld;
  T* crow = reinterpret_cast<T*>(p.cache) + (long long)s * p.seq_stride + (long long)position * p.cld;
  const int n = p.heads + (p.shared ? 0 : p.kv_heads);
  for (int h = warp; h < n; h += kGaThreads / 32) {
    if (h < p.heads) { T* q = row + p.q_off + (long long)h * p.dim; norm_turn(q, q, p.q_norm, position, lane); }
    else { const int g = h - p.heads; norm_turn(row + p.k_off + (long long)g * p.dim, crow + (long long)g * p.dim, p.k_norm, position, lane); }
  }
  if (p.shared) return;
  if constexpr (PAIRED) {                // in words: the columns of all heads lie side by side in both
    for (int i = threadIdx.x; i < p.kv_heads * p.vdim / 2; i += kGaThreads) reinterpret_cast<uint32_t*>(crow + p.v_col)[i] = reinterpret_cast<const uint32_t*>(row + p.v_off)[i];
  } else {
    for (int i = threadIdx.x; i < p.kv_heads * p.vdim; i += kGaThreads) crow[p.v_col + i] = row[p.v_off + i];
  }
}
Status grouped_append(cudaStream_t s, const GroupedAttnDesc& d) {
  GaParams p;
  AG_RETURN_IF_ERROR(ga_params(d, &p));
  auto on = [](const void* q, uintptr_t n) { return (reinterpret_cast<uintptr_t>(q) & (n - 1)) == 0; };
  p.paired = d.dtype != DType::F32 && 2 * p.pairs == p.dim && p.pairs % 2 == 0 && p.pairs <= 128 && p.ld % 2 == 0 && p.q_off % 2 == 0 && (p.shared || (p.k_off % 2 == 0 && p.v_off % 2 == 0)) &&
             p.cld % 2 == 0 && p.v_col % 2 == 0 && p.seq_stride % 2 == 0 && p.kv_heads * p.vdim % 2 == 0 && on(p.proj, 4) && on(p.cache, 4) && on(p.q_norm, 8) && on(p.k_norm, 8) && on(p.rot, 16);
  cudaError_t e = cudaSuccess;
  const dim3 grid((unsigned)(d.n_seq * d.T)), block(kGaThreads);
  if (p.paired) e = d.dtype == DType::BF16 ? launch_pdl(grouped_append_kernel<__nv_bfloat16, true>, grid, block, 0, s, p) : launch_pdl(grouped_append_kernel<__half, true>, grid, block, 0, s, p);
  else AG_DISPATCH_FLOAT(d.dtype, T, (e = launch_pdl(grouped_append_kernel<T, false>, grid, block, 0, s, p)));
  return cuda_status(e, "grouped append");
}

// ── decode ──────────────────────────────────────────────────────────────────
constexpr int kGdSplits = 8;                         // CTAs of a cluster at most
constexpr int kGdKeys = 64, kGdOut = 8;              // keys per tile; accumulators per thread: heads * vdim <= 256 * kGdOut
static int gd_pitch(int n, size_t esz) { const int per = 16 / (int)esz, q = (n + per - 1) / per; return (q % 2 ? q : q + 1) * per; }   // an odd number of 16-byte pieces

template <typename T, int NO>
__global__ void __launch_bounds__(256) grouped_decode_kernel(const GaParams p, int kp, int vp) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  constexpr int N = Pack<T>::N;
  T* sk = reinterpret_cast<T*>(smem_raw);                          // [kGdKeys][kp]
  T* sv = sk + kGdKeys * kp;                                       // [kGdKeys][vp]
  float* sq = reinterpret_cast<float*>(sv + kGdKeys * vp);         // [hg][kp], zero past dim
  float* sp = sq + p.hg * kp;                                      // [hg][kGdKeys]
  float* s_m = sp + p.hg * kGdKeys;                                // [hg] maximum, sum, rescale factor
  float* s_l = s_m + p.hg;
  float* s_a = s_l + p.hg;
  float* so = s_a + p.hg;                                          // [hg][vdim] of this split
  const int split = (int)sm100::cluster_ctarank(), splits = (int)gridDim.x;
  const int kh = (int)blockIdx.y / p.h_parts, part = (int)blockIdx.y % p.h_parts, h0 = kh * p.group + part * p.hg, nh = min(p.hg, p.group - part * p.hg);
  const int r = blockIdx.z, s = r / p.T, t = r % p.T, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Positions and the rows below them are older than the launch before this one, which has appended this portion's rows and waited for
  // its own predecessor ahead of letting this one start: they are read before the dependency wait.
  const int old_rows = p.pos[s], last = min(old_rows + t + 1, p.max_len), from = p.window ? max(0, last - p.window) : 0;
  const int per = ((last - from + splits - 1) / splits + 7) / 8 * 8;
  const int k_lo = min(last, from + split * per), k_hi = min(last, k_lo + per);
  const T* Q = reinterpret_cast<const T*>(p.proj) + (long long)r * p.ld + p.q_off + (long long)h0 * p.dim;
  const T* K = reinterpret_cast<const T*>(p.cache) + (long long)s * p.seq_stride + (long long)kh * p.dim;
  const T* V = reinterpret_cast<const T*>(p.cache) + (long long)s * p.seq_stride + p.v_col + (long long)kh * p.vdim;
  const bool kvec = p.dim % N == 0, vvec = p.vdim % N == 0;        // rows of a head then start on 16 bytes
  // rows k0 + [0, kGdKeys) that lie in [lo, hi) into shared memory: neighbouring lanes take a row's pieces
  auto stage = [&](T* dst, int pitch, const T* src, int n, bool vec, int k0, int lo, int hi) {
    if (vec) {
      const int q = n / N, rows = 256 / q;                         // q <= 256 pieces where a head fits
      const int j0 = q <= 256 ? (int)threadIdx.x / q : 0, c0 = q <= 256 ? (int)threadIdx.x % q : (int)threadIdx.x;
      if (q <= 256 && j0 >= rows) return;
      for (int j = j0; j < kGdKeys; j += q <= 256 ? rows : 1) {
        if (k0 + j < lo || k0 + j >= hi) continue;
        for (int c = c0; c < q; c += q <= 256 ? q : 256)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm100::smem_u32(dst + j * pitch + c * N)), "l"(src + (long long)(k0 + j) * p.cld + c * N));
      }
    } else {
      const int q = (n + N - 1) / N * N;
      for (int i = threadIdx.x; i < kGdKeys * q; i += 256) {
        const int j = i / q, c = i % q;
        if (k0 + j >= lo && k0 + j < hi) dst[j * pitch + c] = c < n ? src[(long long)(k0 + j) * p.cld + c] : Cvt<T>::from(0.f);
      }
    }
  };
  auto stage_both = [&](int k0, int lo, int hi) { stage(sk, kp, K, p.dim, kvec, k0, lo, hi); stage(sv, vp, V, p.vdim, vvec, k0, lo, hi); };
  stage_both(k_lo, k_lo, min(k_hi, old_rows));
  pdl_wait();
  pdl_trigger();
  for (int i = threadIdx.x; i < p.hg * kp; i += 256) { const int hh = i / kp, c = i % kp; sq[i] = hh < nh && c < p.dim ? Cvt<T>::to(Q[(long long)hh * p.dim + c]) * p.scale : 0.f; }
  if (threadIdx.x < p.hg) { s_m[threadIdx.x] = -INFINITY; s_l[threadIdx.x] = 0.f; }
  float acc[NO];
#pragma unroll
  for (int n = 0; n < NO; n++) acc[n] = 0.f;
  const int outs = nh * p.vdim;
  const int kpacks = (p.dim + N - 1) / N;
  for (int k0 = k_lo; k0 < k_hi; k0 += kGdKeys) {
    const int nk = min(kGdKeys, k_hi - k0);
    if (k0 != k_lo) __syncthreads();
    stage_both(k0, k0 == k_lo ? max(k0, old_rows) : k0, k_hi);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int key = threadIdx.x & (kGdKeys - 1);
    for (int hh = threadIdx.x / kGdKeys; hh < nh; hh += 256 / kGdKeys) {
      float a = -INFINITY;
      if (key < nk) {
        float part[4] = {0.f, 0.f, 0.f, 0.f};          // four chains: a column waits for the one four before it
#pragma unroll 2
        for (int q = 0; q < kpacks; q++) {
          const Pack<T> kv = *reinterpret_cast<const Pack<T>*>(sk + key * kp + q * N);
          const float* qv = sq + hh * kp + q * N;
#pragma unroll
          for (int e = 0; e < N; e++) part[e & 3] = fmaf(qv[e], Cvt<T>::to(kv.v[e]), part[e & 3]);
        }
        a = (part[0] + part[1]) + (part[2] + part[3]);
        if (p.cap > 0.f) a = p.cap * tanhf(a / p.cap);
      }
      sp[hh * kGdKeys + key] = a;
    }
    __syncthreads();
    for (int hh = warp; hh < nh; hh += 8) {
      const float x0 = sp[hh * kGdKeys + lane], x1 = sp[hh * kGdKeys + lane + 32];
      const float m0 = s_m[hh], m1 = fmaxf(m0, warp_max(fmaxf(x0, x1)));
      const float e0 = x0 == -INFINITY ? 0.f : expf(x0 - m1), e1 = x1 == -INFINITY ? 0.f : expf(x1 - m1);
      const float sum = warp_sum(e0 + e1);
      sp[hh * kGdKeys + lane] = e0; sp[hh * kGdKeys + lane + 32] = e1;
      __syncwarp();
      if (lane == 0) { const float a = m0 == -INFINITY ? 0.f : expf(m0 - m1); s_a[hh] = a; s_l[hh] = s_l[hh] * a + sum; s_m[hh] = m1; }
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NO; n++) {
      const int o = threadIdx.x + n * 256;
      if (o < outs) {
        const int hh = o / p.vdim, c = o % p.vdim;
        float a = acc[n] * s_a[hh];
        const float* w = sp + hh * kGdKeys;
#pragma unroll 8
        for (int j = 0; j < nk; j++) a = fmaf(w[j], Cvt<T>::to(sv[j * vp + c]), a);
        acc[n] = a;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int n = 0; n < NO; n++) { const int o = threadIdx.x + n * 256; if (o < outs) so[o] = acc[n]; }
  if (splits > 1) sm100::cluster_sync_all(); else __syncthreads();
  // every CTA finishes a share of the outputs
  auto remote = [&](const float* x, int q) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(sm100::mapa_u32(sm100::smem_u32(x), (uint32_t)q)));
    return v;
  };
  T* y = reinterpret_cast<T*>(p.y) + (long long)r * p.y_ld + (long long)h0 * p.vdim;
  for (int o = split * 256 + threadIdx.x; o < outs; o += splits * 256) {
    const int hh = o / p.vdim;
    float m = -INFINITY, l = 0.f, a = 0.f, mq[kGdSplits], lq[kGdSplits], aq[kGdSplits];
#pragma unroll
    for (int q = 0; q < kGdSplits; q++) {              // all of the cluster's at once
      mq[q] = q < splits ? remote(s_m + hh, q) : -INFINITY;
      lq[q] = q < splits ? remote(s_l + hh, q) : 0.f;
      aq[q] = q < splits ? remote(so + o, q) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < kGdSplits; q++) m = fmaxf(m, mq[q]);
#pragma unroll
    for (int q = 0; q < kGdSplits; q++) {
      if (mq[q] == -INFINITY) continue;
      const float f = expf(mq[q] - m);
      l = fmaf(f, lq[q], l);
      a = fmaf(f, aq[q], a);
    }
    y[o] = Cvt<T>::from(a / l);
  }
  if (splits > 1) sm100::cluster_sync_all();        // no CTA leaves while its sums are being read
}

template <typename T, int NO>
static cudaError_t launch_gd(cudaStream_t s, const GaParams& p, int splits, int kp, int vp, size_t smem) {
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(grouped_decode_kernel<T, NO>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)splits, (unsigned)(p.kv_heads * p.h_parts), (unsigned)(p.n_seq * p.T)); cfg.blockDim = dim3(256); cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension; at[1].val.clusterDim.x = (unsigned)splits; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, grouped_decode_kernel<T, NO>, p, kp, vp);
}

Status grouped_decode(cudaStream_t s, const GroupedAttnDesc& d) {
  GaParams p;
  AG_RETURN_IF_ERROR(ga_params(d, &p));
  if (!d.y || !aligned16(d.cache) || d.seq_stride % 8) return Status::invalid("grouped decode: missing or misaligned operand");
  if (d.vdim > 256 * kGdOut || p.kv_heads > 65535 / p.group || d.n_seq * d.T > 65535) return Status::unsupported("grouped decode: heads too large or too many");
  p.hg = std::min({p.group, 8, 256 * kGdOut / d.vdim});
  p.h_parts = (p.group + p.hg - 1) / p.hg;
  // splits: a cluster of up to eight; about a tile of keys each at least, and no more than fill the machine twice
  const int reach = d.window ? std::min(d.window, d.max_len) : d.max_len;
  int splits = 1;
  while (splits < kGdSplits && splits * 2 * 32 <= reach && splits * p.kv_heads * p.h_parts * d.n_seq * d.T < 2 * sm_count()) splits *= 2;
  cudaError_t e = cudaSuccess;
  AG_DISPATCH_FLOAT(d.dtype, T, {
    const int kp = gd_pitch(d.dim, sizeof(T)), vp = gd_pitch(d.vdim, sizeof(T));
    const size_t smem = (size_t)kGdKeys * (kp + vp) * sizeof(T) + ((size_t)p.hg * kp + (size_t)p.hg * kGdKeys + 3 * p.hg + (size_t)p.hg * d.vdim) * sizeof(float);
    if (smem > 220 * 1024) return Status::unsupported("grouped decode: head too large");
    const int no = (p.hg * d.vdim + 255) / 256;
    if (no <= 1) e = launch_gd<T, 1>(s, p, splits, kp, vp, smem);
    else if (no <= 2) e = launch_gd<T, 2>(s, p, splits, kp, vp, smem);
    else if (no <= 4) e = launch_gd<T, 4>(s, p, splits, kp, vp, smem);
    else e = launch_gd<T, 8>(s, p, splits, kp, vp, smem);
  });
  return cuda_status(e, "grouped decode");
}

}}  // namespace ag::k
