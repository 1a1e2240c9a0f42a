// float32 products on the tensor cores.
//
// Both operands are split into three bf16 planes, x = x0 + x1 + x2 (each the bf16 rounding of what the planes before it left), and
// the six largest cross terms a0 b0, a0 b1, a1 b0, a0 b2, a1 b1, a2 b0 are multiplied by tcgen05 (error about 2^-22 of the product, while
// the third plane of what matters lies in bf16's range: an operand below 2^-117, 6e-36, keeps 2^-133 absolute, which a factor of 1e30 in
// the other operand can bring to light). What is not finite in the sum of a0 b0 is the result as it stands: an infinity has no other
// planes, and what it makes of the other operand's is not looked at. So infinities and NaN come out as float32 sums have them, at no cost
// in time. A finite number that bf16 rounds to an infinity (0.2 % below the largest float32) is noted by the pass that writes the planes;
// then the results that are not finite are taken again in float32, a warp to a result.
// A pipeline stage holds the three planes of one 64-deep k-block of A and B, and its six products run from that one copy: 72 KB per
// 24 MMAs and CTA, where a GEMM over a six-fold K extent (what this replaces) fetches 12 tiles for the same work, and the planes are
// written once instead of each term as often as a product names it (10 bytes per element moved instead of 16).
// The tensor core truncates where it adds, so a long accumulation drifts (K = 768 in one go: 7.3e-7 of the result's norm off, all of it
// towards zero, against 5.0e-7 for the CUDA-core kernel's rounded sums). a0 b0 therefore has an accumulator of its own, and no
// accumulation runs over more than kF3Chunk k-blocks: the epilogue warps add the chunks up in registers, rounded to nearest, under the
// next chunk's products.
//
// Tiles of 256 x 128 on CTA pairs (cta_group::2), 256 x 256 for large products (f3_wide); with the former two accumulator pairs of 2 x 128 TMEM columns, so the epilogue of a tile runs under the
// next one's products. A product with few tiles also splits K: each share is one unit of the persistent grid, leaves its sum in
// a workspace, and a second kernel adds the shares in K order and applies the epilogue.
//
// Bound: shared-memory bandwidth beside the tensor pipe (a 256 x 128 tile reads 96 to 128 bytes a clock and SM for its operands): about 2 250
// cycles a k-block against 1 536 at the tensor rate; sm__pipe_tensor_cycles_active 68 % on 1024 x 50257 x 768. Before -> after in a GPT-2-small
// forward of 1024 rows, us: the 48 linears 2 910 -> 1 370 with 93 for the shares, LM head 519 -> 339, planes 555 -> 397, whole 4 430 -> 2 690.
#include "common.cuh"
#include "sm100.cuh"
#include <algorithm>
#include <atomic>
#include <cmath>

namespace ag { namespace k {
using namespace sm100;

Status make_map(CUtensorMap* out, DType dt, const void* ptr, uint64_t inner, uint64_t rows, uint64_t nbi, uint64_t nbo, uint64_t row_stride, uint64_t bi_stride,
                uint64_t bo_stride, uint32_t b0, uint32_t b1);
int* matmul_status_word();

// ── planes ──────────────────────────────────────────────────────────────────
struct PlaneJob { const float* in; __nv_bfloat16* out; long long rows, cols, row_stride, batch_stride; int batches, blocks; };

__global__ void __launch_bounds__(256) f32_planes_kernel(const __grid_constant__ PlaneJob ja, const __grid_constant__ PlaneJob jb, unsigned long long* note, unsigned long long call) {
  pdl_wait();
  pdl_trigger();
  const bool second = (int)blockIdx.x >= ja.blocks;
  const PlaneJob& j = second ? jb : ja;
  const long long packs = j.cols / 8, plane = j.rows * j.cols, per = j.rows * packs, total = per * j.batches;
  const long long step = (long long)j.blocks * 256;
  bool noted = false;
  for (long long i = (long long)(blockIdx.x - (second ? ja.blocks : 0)) * 256 + threadIdx.x; i < total; i += step) {
    const long long b = j.batches > 1 ? i / per : 0, q = i - b * per, r = q / packs, c = (q - r * packs) * 8;
    const float* src = j.in + b * j.batch_stride + r * j.row_stride + c;
    const float4 x0 = __ldcs(reinterpret_cast<const float4*>(src)), x1 = __ldcs(reinterpret_cast<const float4*>(src + 4));
    const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    Pack<__nv_bfloat16> t[3];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const __nv_bfloat16 h0 = __float2bfloat16_rn(x[e]);
      const float r1 = x[e] - __bfloat162float(h0);
      const __nv_bfloat16 h1 = __float2bfloat16_rn(r1);
      const float r2 = r1 - __bfloat162float(h1);
      t[0].v[e] = h0; t[1].v[e] = h1; t[2].v[e] = __float2bfloat16_rn(r2);
    }
    const uint4 w = *reinterpret_cast<const uint4*>(&t[0]);
    auto odd = [](uint32_t u) { return (u & 0x7f807f80u) + 0x00800080u; };                     // bits 15 and 31: an exponent of ones
    if ((odd(w.x) | odd(w.y) | odd(w.z) | odd(w.w)) & 0x80008000u) {
#pragma unroll
      for (int e = 0; e < 8; e++) {
        if (isfinite(__bfloat162float(t[0].v[e]))) continue;
        noted |= isinf(__bfloat162float(t[1].v[e]));                                           // a finite number less an infinity
        t[1].v[e] = __float2bfloat16_rn(0.f); t[2].v[e] = t[1].v[e];
      }
    }
    __nv_bfloat16* dst = j.out + b * 3 * plane + r * j.cols + c;
#pragma unroll
    for (int k = 0; k < 3; k++) st16(dst + k * plane, t[k]);
  }
  if (noted) *note = call;
}

// ── the product ─────────────────────────────────────────────────────────────
constexpr int kF3Bm = 128, kF3Bn = 128, kF3Bk = 64, kF3Stages = 3, kF3EpiWarps = 8, kF3Threads = 64 + 32 * kF3EpiWarps;
constexpr int kF3ATile = kF3Bm * kF3Bk * 2, kF3BTile = (kF3Bn / 2) * kF3Bk * 2;      // one plane: this CTA's rows of A, its half of B's columns
constexpr int kF3Stage = 3 * (kF3ATile + kF3BTile);
constexpr int kF3Chunk = 4;                                                          // k-blocks per accumulation
constexpr int kF3StgPitch = 9;                                                       // floats: 32 rows x 8 columns per warp, no bank conflicts
constexpr int kF3Stg = 32 * kF3StgPitch * 4;
constexpr int kF3Smem = kF3Stages * kF3Stage + kF3EpiWarps * kF3Stg + 1024;
static_assert(kF3Smem + 512 <= 232448, "shared memory of a CTA");

struct F3Params {
  float* c; const float* bias; const float* residual; float* partial;
  float alpha; int act, m, n, batch, a_one, b_one, num_kb, tiles_m, tiles_n, splits, kb_per_split, vec;
  long long c_row, c_batch, p_row;
  const float* a; const float* b;        // the operands as they were given; *note == call: one of them holds a finite number beyond bf16
  int k; long long a_row, a_batch, b_row, b_col, b_batch;
  const unsigned long long* note; unsigned long long call;
  int* status;
};

// Out of line: 64 copies of the two GELUs would be most of the kernel's code, fetched anew by every launch.
__device__ __noinline__ float4 f3_act(float4 v, int act) {
  switch ((Act)act) {
    case Act::GeluTanh: return make_float4(gelu_tanh_f(v.x), gelu_tanh_f(v.y), gelu_tanh_f(v.z), gelu_tanh_f(v.w));
    case Act::GeluErf: return make_float4(gelu_erf_f(v.x), gelu_erf_f(v.y), gelu_erf_f(v.z), gelu_erf_f(v.w));
    case Act::Relu: return make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f));
    default: return v;
  }
}

// n neighbouring results of each lane's row, of which those that are not finite are taken again; a warp adds one up. The other warps wait two
// seconds at most for the epilogue's, so there a call takes `most` results (kF3Again; all of them up to K = 8192) and reports any beyond:
// at 92 cycles of an SM for 32 of K, a tile's eight warps with four calls each take half a second.
constexpr int kF3Again = 1 << 23;         // times K
__device__ __forceinline__ bool f3_again(const F3Params& p) { return __ldcg(p.note) == p.call; }
__device__ __noinline__ void f3_plain(const F3Params& p, bool in, int b, long long row, int col0, int n, float* v, int most) {
  const int lane = threadIdx.x & 31;
  for (int e = 0; e < n; e++) {
    for (unsigned again = __ballot_sync(0xffffffffu, in && col0 + e < p.n && !isfinite(v[e])); again; again &= again - 1) {
      if (most-- == 0) { if (lane == 0) atomicCAS(p.status, 0, 9); return; }
      const int who = __ffs(again) - 1;
      const float* a = p.a + __shfl_sync(0xffffffffu, b, who) * p.a_batch + __shfl_sync(0xffffffffu, row, who) * p.a_row;
      const float* w = p.b + __shfl_sync(0xffffffffu, b, who) * p.b_batch + (__shfl_sync(0xffffffffu, col0, who) + e) * p.b_col;
      float t = 0.f;
#pragma unroll 4
      for (int i = lane; i < p.k; i += 32) t = fmaf(__ldg(a + i), __ldg(w + i * p.b_row), t);
      t = warp_sum(t);
      if (lane == who) v[e] = t;
    }
  }
}

// Epilogue of 32 columns: a lane has its row's.
__device__ __forceinline__ void f3_store(const F3Params& p, float (&v)[32], int b, long long row0, int col0, float bias_l, float* stg) {
  const int lane = threadIdx.x & 31;
  const long long gm = row0 + lane;
  bool odd = false;
#pragma unroll
  for (int e = 0; e < 32; e++) odd |= !isfinite(v[e]);
  if (__any_sync(0xffffffffu, odd) && f3_again(p)) {
    float t[32];
#pragma unroll
    for (int e = 0; e < 32; e++) t[e] = v[e];
    f3_plain(p, gm < p.m, b, gm, col0, 32, t, kF3Again / p.k);
#pragma unroll
    for (int e = 0; e < 32; e++) v[e] = t[e];
  }
  __syncwarp();
#pragma unroll
  for (int e = 0; e < 32; e++) v[e] = fmaf(v[e], p.alpha, __shfl_sync(0xffffffffu, bias_l, e));
  if (p.act) {
#pragma unroll
    for (int e = 0; e < 32; e += 4) {
      const float4 o = f3_act(make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]), p.act);
      v[e] = o.x; v[e + 1] = o.y; v[e + 2] = o.z; v[e + 3] = o.w;
    }
  }
  const long long at = (long long)b * p.c_batch + row0 * p.c_row + col0;
  if (p.vec && col0 + 32 <= p.n) {
    if (gm < p.m) {
      float* crow = p.c + at + lane * p.c_row;
      const float* rrow = p.residual ? p.residual + at + lane * p.c_row : nullptr;
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        float4 o = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
        if (rrow) { const float4 r = *reinterpret_cast<const float4*>(rrow + e); o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w; }
        *reinterpret_cast<float4*>(crow + e) = o;
      }
    }
    return;
  }
  // rows on any 4-byte boundary, or a ragged column block: four rows of eight columns per store instead of 32 rows of one
#pragma unroll
  for (int e0 = 0; e0 < 32; e0 += 8) {
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; e++) stg[lane * kF3StgPitch + e] = v[e0 + e];
    __syncwarp();
    const int c = lane & 7, col = col0 + e0 + c;
#pragma unroll
    for (int r = lane >> 3; r < 32; r += 4) {
      if (row0 + r < p.m && col < p.n) {
        const long long o = at + r * p.c_row + e0 + c;
        const float x = stg[r * kF3StgPitch + c];
        p.c[o] = p.residual ? x + p.residual[o] : x;
      }
    }
  }
}

// One MMA of a CTA pair whose descriptors differ from one another in their low words only. 24 of them take 1 536 cycles of a
// k-block, so the issuing thread has 64 cycles for each: the words are sums with constants, nothing is packed in 64 bits.
__device__ __forceinline__ void f3_mma(uint32_t d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n setp.ne.b32 p, %6, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %5, p;\n}"
      ::"r"(d), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate) : "memory");
}

template <bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kF3Threads, 1)
gemm_f32x3_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ F3Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[kF3Stages], empty_bar[kF3Stages], tmem_full_bar[2], tmem_empty_bar[2];
  __shared__ uint32_t tmem_base_slot;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int tiles = p.tiles_m * p.tiles_n;
  const long long units = (long long)tiles * p.batch * p.splits, first = blockIdx.x >> 1, step = gridDim.x >> 1;
  // unit -> share of K (outermost), batch entry, column block, row block (innermost: neighbours share B)
  auto unit = [&](long long u, int& m0, int& n0, int& b, int& kb0, int& kb1, int& split) {
    const long long t = u % ((long long)tiles * p.batch);
    split = (int)(u / ((long long)tiles * p.batch));
    b = (int)(t / tiles);
    const int rem = (int)(t % tiles);
    m0 = (rem % p.tiles_m) * 2 * kF3Bm + (int)rank * kF3Bm;
    n0 = rem / p.tiles_m * kF3Bn;
    kb0 = split * p.kb_per_split;
    kb1 = min(p.num_kb, kb0 + p.kb_per_split);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kF3Stages; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int a = 0; a < 2; a++) { mbar_init(&tmem_full_bar[a], 1); mbar_init(&tmem_empty_bar[a], 2 * kF3EpiWarps); }
    mbar_fence_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_slot, 512); tmem_relinquish_pair(); }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_wait();
  pdl_trigger();
  int m0, n0, b, kb0, kb1, split;

  if (warp == 0) {
    if (lane == 0) {                                   // loads (both CTAs; the even CTA's barriers count the bytes of both)
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (long long u = first; u < units && ok; u += step) {
        unit(u, m0, n0, b, kb0, kb1, split);
        const int nh = n0 + (int)rank * (kF3Bn / 2), ba = p.a_one ? 0 : b, bb = p.b_one ? 0 : b;
        for (int kb = kb0; kb < kb1; kb++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, p.status, 1)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * kF3Stage);
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), 0);
          uint8_t* sa = smem + stage * kF3Stage;
          uint8_t* sb = sa + 3 * kF3ATile;
#pragma unroll
          for (int q = 0; q < 3; q++) {
            tma_load_4d_pair(sa + q * kF3ATile, &tmap_a, bar, kb * kF3Bk, m0, q, ba);
            if (B_MN) tma_load_4d_pair(sb + q * kF3BTile, &tmap_b, bar, nh, kb * kF3Bk, q, bb);
            else tma_load_4d_pair(sb + q * kF3BTile, &tmap_b, bar, kb * kF3Bk, nh, q, bb);
          }
          if (++stage == kF3Stages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {                      // products
      constexpr uint32_t idesc = make_idesc_f16(1, 0, B_MN ? 1 : 0, 2 * kF3Bm, kF3Bn);
      int stage = 0, acc = 0; uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (long long u = first; u < units && ok; u += step) {
        unit(u, m0, n0, b, kb0, kb1, split);
        for (int kc = kb0; kc < kb1 && ok; kc += kF3Chunk) {
          if (!mbar_wait(&tmem_empty_bar[acc], acc_phase ^ 1, p.status, 2)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t d_hi = tmem_base + (uint32_t)(acc * 256), d_lo = d_hi + 128;
          for (int kb = kc; kb < min(kb1, kc + kF3Chunk); kb++) {
            if (!mbar_wait(&full_bar[stage], phase, p.status, 3)) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t sa = smem_u32(smem + stage * kF3Stage);
            const uint64_t a0 = make_smem_desc_sw128(sa, 16, 1024), b0 = make_smem_desc_sw128(sa + 3 * kF3ATile, B_MN ? 64 * 128 : 16, 1024);
            const uint32_t ah = (uint32_t)(a0 >> 32), bh = (uint32_t)(b0 >> 32), al = (uint32_t)a0, bl = (uint32_t)b0;
            uint32_t on = kb > kc ? 1u : 0u;
#pragma unroll
            for (int kk = 0; kk < kF3Bk / 16; kk++) {
              auto mma = [&](uint32_t d, int qa, int qb, uint32_t acc_on) {
                f3_mma(d, al + (uint32_t)((qa * kF3ATile + kk * 32) >> 4), ah, bl + (uint32_t)((qb * kF3BTile + kk * (B_MN ? 16 * 128 : 32)) >> 4), bh, idesc, acc_on);
              };
              mma(d_lo, 2, 0, on);
              mma(d_lo, 1, 1, 1u);
              mma(d_lo, 0, 2, 1u);
              mma(d_lo, 1, 0, 1u);
              mma(d_lo, 0, 1, 1u);
              mma(d_hi, 0, 0, on);
              on = 1u;
            }
            mma_commit_both(&empty_bar[stage]);
            if (++stage == kF3Stages) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          mma_commit_both(&tmem_full_bar[acc]);
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
  } else {                                             // epilogue: a warp has 32 rows of its CTA and 64 of the tile's columns
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float* stg = reinterpret_cast<float*>(smem + kF3Stages * kF3Stage) + (warp - 2) * (32 * kF3StgPitch);
    int acc = 0; uint32_t acc_phase = 0;
    bool ok = true;
    for (long long u = first; u < units; u += step) {
      unit(u, m0, n0, b, kb0, kb1, split);
      const long long row0 = m0 + quarter * 32, gm = row0 + lane;
      float bias_l[2];
#pragma unroll
      for (int g = 0; g < 2; g++) {
        const int col = n0 + half * 64 + g * 32 + lane;
        bias_l[g] = p.bias && !p.partial && col < p.n ? __ldg(p.bias + col) : 0.f;
      }
      float sum[2][32];
#pragma unroll
      for (int g = 0; g < 2; g++)
#pragma unroll
        for (int e = 0; e < 32; e++) sum[g][e] = 0.f;
      for (int kc = kb0; kc < kb1; kc += kF3Chunk) {
        if (!__all_sync(0xffffffffu, mbar_wait(&tmem_full_bar[acc], acc_phase, p.status, 4))) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * 256 + half * 64);
#pragma unroll
        for (int g = 0; g < 2; g++) {
          uint32_t hi[32], lo[32];
          tmem_ld_32x32(taddr + g * 32, hi);
          tmem_ld_32x32(taddr + 128 + g * 32, lo);
          tmem_ld_wait();
          float odd = 0.f;
#pragma unroll
          for (int e = 0; e < 32; e++) {
            const float x = __uint_as_float(hi[e]) + __uint_as_float(lo[e]);
            odd = fmaf(x, 0.f, odd);
            lo[e] = __float_as_uint(x);
          }
          if (odd != odd) {                            // something is not finite: the sum of a0 b0 as it stands
#pragma unroll
            for (int e = 0; e < 32; e++) if (!isfinite(__uint_as_float(hi[e]))) lo[e] = hi[e];
          }
#pragma unroll
          for (int e = 0; e < 32; e++) sum[g][e] += __uint_as_float(lo[e]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty_bar[acc]), 0));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (!ok) break;
#pragma unroll
      for (int g = 0; g < 2; g++) {
        const int col0 = n0 + half * 64 + g * 32;
        if (row0 >= p.m || col0 >= p.n) continue;      // uniform across the warp
        float (&v)[32] = sum[g];
        if (p.partial) {
          float* dst = p.partial + ((long long)(split * p.batch + b) * p.m + gm) * p.p_row + col0;
          if (gm < p.m) {
#pragma unroll
            for (int e = 0; e < 32; e += 4) if (col0 + e < p.n) *reinterpret_cast<float4*>(dst + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
          }
          continue;
        }
        f3_store(p, v, b, row0, col0, bias_l[g], stg);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();      // neither CTA leaves while its peer can still signal its barriers or run MMAs on its shared memory
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ── tiles of 256 x 256 ──────────────────────────────────────────────────────
// A third fewer operand reads per product than in the kernel above, for products that are long in every direction. TMEM then has room for
// one accumulator of each kind (2 x 256 columns): a0 b0, the first product of a k-block, is drained under the block's small ones, and
// those, every kFwLowChunk blocks, under the next a0 b0. A slot of the ring is one plane of a k-block's A and B (32 KB), planes in the
// order 1, 0, 2. Two blocks of a0 b0 in an accumulation leave less truncation than four do (4096^3: 1.6e-7 of the norm off, 2.4e-7 in the
// kernel above); small products drained as often would cost more in rounded additions than they lose to truncation.
// What bounds it is the power limit: 8 x 4096^3 takes 4 880 us with the planes' 400, 1.47 PFLOP/s of bf16 products (sustained rate of one
// plain bf16 product of 8192^3: 1.44).
constexpr int kFwBn = 256, kFwSlots = 6, kFwTile = kF3Bm * kF3Bk * 2, kFwSlot = 2 * kFwTile;
constexpr int kFwSmem = kFwSlots * kFwSlot + kF3EpiWarps * kF3Stg + 1024;
constexpr int kFwChunk = 2, kFwLowChunk = 16;            // k-blocks in one accumulation of a0 b0, of the small products
static_assert(kFwLowChunk % kFwChunk == 0, "the two drains meet");
constexpr int kFwBand = 8;                // row blocks that share a walk over the column blocks
static_assert(kFwSmem + 512 <= 232448, "shared memory of a CTA");

template <bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kF3Threads, 1)
gemm_f32x3_wide_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ F3Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full_bar[kFwSlots], empty_bar[kFwSlots], hi_full, hi_empty, lo_full, lo_empty;
  __shared__ uint32_t tmem_base_slot;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int tiles = p.tiles_m * p.tiles_n;
  const long long units = (long long)tiles * p.batch, first = blockIdx.x >> 1, step = gridDim.x >> 1;
  auto unit = [&](long long u, int& m0, int& n0, int& b) {
    b = (int)(u / tiles);
    const int t = (int)(u % tiles), band = t / (kFwBand * p.tiles_n), r = t - band * kFwBand * p.tiles_n, high = min(kFwBand, p.tiles_m - band * kFwBand);
    m0 = (band * kFwBand + r % high) * 2 * kF3Bm + (int)rank * kF3Bm;
    n0 = r / high * kFwBn;
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFwSlots; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&hi_full, 1); mbar_init(&lo_full, 1);
    mbar_init(&hi_empty, 2 * kF3EpiWarps); mbar_init(&lo_empty, 2 * kF3EpiWarps);
    mbar_fence_init();
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) { tmem_alloc_pair(&tmem_base_slot, 512); tmem_relinquish_pair(); }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after_sync();
  const uint32_t tmem_base = tmem_base_slot;
  pdl_wait();
  pdl_trigger();
  int m0, n0, b;

  if (warp == 0) {
    if (lane == 0) {                                   // loads
      int slot = 0; uint32_t phase = 0;
      bool ok = true;
      for (long long u = first; u < units && ok; u += step) {
        unit(u, m0, n0, b);
        const int nh = n0 + (int)rank * (kFwBn / 2), ba = p.a_one ? 0 : b, bb = p.b_one ? 0 : b;
        for (int kb = 0; kb < p.num_kb && ok; kb++) {
          for (int i = 0; i < 3; i++) {
            const int q = i == 2 ? 2 : 1 - i;
            if (!mbar_wait(&empty_bar[slot], phase ^ 1, p.status, 5)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(&full_bar[slot], 2 * kFwSlot);
            const uint32_t bar = mapa_u32(smem_u32(&full_bar[slot]), 0);
            uint8_t* sa = smem + slot * kFwSlot;
            uint8_t* sb = sa + kFwTile;
            tma_load_4d_pair(sa, &tmap_a, bar, kb * kF3Bk, m0, q, ba);
#pragma unroll
            for (int h = 0; h < 2; h++) {
              if (B_MN) tma_load_4d_pair(sb + h * (kFwTile / 2), &tmap_b, bar, nh + h * 64, kb * kF3Bk, q, bb);
              else tma_load_4d_pair(sb + h * (kFwTile / 2), &tmap_b, bar, kb * kF3Bk, nh + h * 64, q, bb);
            }
            if (++slot == kFwSlots) { slot = 0; phase ^= 1; }
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {                      // products
      constexpr uint32_t idesc = make_idesc_f16(1, 0, B_MN ? 1 : 0, 2 * kF3Bm, kFwBn);
      const uint64_t a0 = make_smem_desc_sw128(smem_u32(smem), 16, 1024), b0 = make_smem_desc_sw128(smem_u32(smem) + kFwTile, B_MN ? 64 * 128 : 16, 1024);
      const uint32_t ah = (uint32_t)(a0 >> 32), bh = (uint32_t)(b0 >> 32), al = (uint32_t)a0, bl = (uint32_t)b0;
      const uint32_t d_hi = tmem_base, d_lo = tmem_base + 256;
      auto products = [&](uint32_t d, int slot_a, int slot_b, uint32_t on) {
#pragma unroll
        for (int kk = 0; kk < kF3Bk / 16; kk++)
          f3_mma(d, al + (uint32_t)((slot_a * kFwSlot + kk * 32) >> 4), ah, bl + (uint32_t)((slot_b * kFwSlot + kk * (B_MN ? 16 * 128 : 32)) >> 4), bh, idesc, kk ? 1u : on);
      };
      int slot = 0; uint32_t phase = 0, hi_phase = 0, lo_phase = 0;
      auto next = [&]() { const int s = slot; if (++slot == kFwSlots) { slot = 0; phase ^= 1; } return s; };
      auto arrived = [&]() {
        const bool here = mbar_wait(&full_bar[slot], phase, p.status, 7);
        tc_fence_after_sync();
        return here;
      };
      bool ok = true;
      for (long long u = first; u < units && ok; u += step) {
        for (int kb = 0; kb < p.num_kb; kb++) {
          if (!arrived()) { ok = false; break; }
          const int s1 = next();
          if (!arrived()) { ok = false; break; }
          const int s0 = next();
          if (kb % kFwChunk == 0) {
            if (!mbar_wait(&hi_empty, hi_phase ^ 1, p.status, 6)) { ok = false; break; }
            hi_phase ^= 1;
            tc_fence_after_sync();
          }
          products(d_hi, s0, s0, kb % kFwChunk ? 1u : 0u);
          if (kb % kFwChunk == kFwChunk - 1 || kb + 1 == p.num_kb) mma_commit_both(&hi_full);
          if (kb % kFwLowChunk == 0) {
            if (!mbar_wait(&lo_empty, lo_phase ^ 1, p.status, 6)) { ok = false; break; }
            lo_phase ^= 1;
            tc_fence_after_sync();
          }
          products(d_lo, s1, s1, kb % kFwLowChunk ? 1u : 0u);
          products(d_lo, s1, s0, 1u);
          products(d_lo, s0, s1, 1u);
          mma_commit_both(&empty_bar[s1]);
          if (!arrived()) { ok = false; break; }
          const int s2 = next();
          products(d_lo, s2, s0, 1u);
          products(d_lo, s0, s2, 1u);
          mma_commit_both(&empty_bar[s0]);
          mma_commit_both(&empty_bar[s2]);
          if (kb % kFwLowChunk == kFwLowChunk - 1 || kb + 1 == p.num_kb) mma_commit_both(&lo_full);
        }
      }
    }
  } else {                                             // epilogue: a warp has 32 rows of its CTA and 128 of the tile's columns
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float* stg = reinterpret_cast<float*>(smem + kFwSlots * kFwSlot) + (warp - 2) * (32 * kF3StgPitch);
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 128);
    uint32_t hi_phase = 0, lo_phase = 0;
    bool ok = true;
    for (long long u = first; u < units; u += step) {
      unit(u, m0, n0, b);
      const long long row0 = m0 + quarter * 32;
      float sum[4][32];
#pragma unroll
      for (int g = 0; g < 4; g++)
#pragma unroll
        for (int e = 0; e < 32; e++) sum[g][e] = 0.f;
      for (int kc = 0; kc < p.num_kb; kc += kFwChunk) {
        if (!__all_sync(0xffffffffu, mbar_wait(&hi_full, hi_phase, p.status, 8))) { ok = false; break; }
        hi_phase ^= 1;
        tc_fence_after_sync();
#pragma unroll
        for (int g = 0; g < 8; g++) {                  // 16 columns at a time: the sums take 128 of 168 registers
          uint32_t hi[16];
          tmem_ld_32x16(taddr + g * 16, hi);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; e++) sum[g / 2][g % 2 * 16 + e] += __uint_as_float(hi[e]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&hi_empty), 0));
        if ((kc + kFwChunk) % kFwLowChunk && kc + kFwChunk < p.num_kb) continue;
        if (!__all_sync(0xffffffffu, mbar_wait(&lo_full, lo_phase, p.status, 8))) { ok = false; break; }
        lo_phase ^= 1;
        tc_fence_after_sync();
#pragma unroll
        for (int g = 0; g < 8; g++) {
          uint32_t lo[16];
          tmem_ld_32x16(taddr + 256 + g * 16, lo);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; e++) if (isfinite(sum[g / 2][g % 2 * 16 + e])) sum[g / 2][g % 2 * 16 + e] += __uint_as_float(lo[e]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&lo_empty), 0));
      }
      if (!ok) break;
#pragma unroll
      for (int g = 0; g < 4; g++) {
        const int col0 = n0 + half * 128 + g * 32;
        if (row0 >= p.m || col0 >= p.n) continue;      // uniform across the warp
        f3_store(p, sum[g], b, row0, col0, p.bias && col0 + lane < p.n ? __ldg(p.bias + col0 + lane) : 0.f, stg);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();      // neither CTA leaves while its peer can still signal its barriers or run MMAs on its shared memory
  tc_fence_after_sync();
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// The shares of K added in order, then what the single-launch epilogue does.
__global__ void __launch_bounds__(256) f32x3_finish_kernel(const __grid_constant__ F3Params p) {
  pdl_wait();
  pdl_trigger();
  const long long q = p.p_row / 4, total = (long long)p.batch * p.m * q, share = (long long)p.batch * p.m * p.p_row;
  const bool look = f3_again(p);
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i - (threadIdx.x & 31) < total; i += (long long)gridDim.x * 256) {      // whole warps
    const bool in = i < total;
    const long long row = min(i, total - 1) / q, col = (min(i, total - 1) - row * q) * 4, b = row / p.m;
    const float* src = p.partial + row * p.p_row + col;
    float4 x[8];
#pragma unroll
    for (int s = 0; s < 8; s++) if (s < p.splits) x[s] = __ldcg(reinterpret_cast<const float4*>(src + s * share));
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 8; s++) if (s < p.splits) { v[0] += x[s].x; v[1] += x[s].y; v[2] += x[s].z; v[3] += x[s].w; }
    const long long at = b * p.c_batch + (row - b * p.m) * p.c_row + col;
    if (look) {
      float t[4] = {v[0], v[1], v[2], v[3]};
      f3_plain(p, in, (int)b, row - b * p.m, (int)col, 4, t, 0x7fffffff);
#pragma unroll
      for (int e = 0; e < 4; e++) v[e] = t[e];
    }
    if (!in) continue;
#pragma unroll
    for (int e = 0; e < 4; e++) v[e] = fmaf(v[e], p.alpha, p.bias && col + e < p.n ? __ldg(p.bias + col + e) : 0.f);
    if (p.act) { const float4 o = f3_act(make_float4(v[0], v[1], v[2], v[3]), p.act); v[0] = o.x; v[1] = o.y; v[2] = o.z; v[3] = o.w; }
    if (p.vec && col + 4 <= p.n) {
      float4 o = make_float4(v[0], v[1], v[2], v[3]);
      if (p.residual) { const float4 r = *reinterpret_cast<const float4*>(p.residual + at); o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w; }
      *reinterpret_cast<float4*>(p.c + at) = o;
    } else {
      for (int e = 0; e < 4 && col + e < p.n; e++) p.c[at + e] = p.residual ? v[e] + p.residual[at + e] : v[e];
    }
  }
}

// Shares of K. A unit of kb k-blocks takes about 1 600 cycles per k-block (24 MMAs of 256 x 128 x 16) and 3 000 around it (first
// loads, last epilogue); splitting costs one more launch and the shares' way through the L2 (about 2 600 bytes per cycle).
int f32x3_splits(int64_t m, int64_t n, int64_t k, int64_t batch) {
  const double pairs = sm_count() / 2, num_kb = (double)((k + kF3Bk - 1) / kF3Bk);
  const double tiles = (double)((m + 2 * kF3Bm - 1) / (2 * kF3Bm)) * (double)((n + kF3Bn - 1) / kF3Bn) * (double)batch;
  int best = 1; double best_cost = 0;
  for (int s = 1; s <= 8; s++) {
    const double kb = std::ceil(num_kb / s);
    if (s > 1 && (kb < 3 || kb * (s - 1) >= num_kb || tiles * s > 4 * pairs)) continue;
    double cost = std::ceil(tiles * s / pairs) * kb * 1600 + 3000;
    if (s > 1) cost += 5000 + (double)m * n * batch * 4 * (2 * s + 1) / 2600;
    if (s == 1 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

// Tiles of 256 x 256 from K = 1024 and three rounds of the grid on. Measured (narrow -> wide, us): 8 x 1536^3 318 -> 306, 16384 x 1024 x 1024
// 224 -> 198, 4096^3 648 -> 643, 8 x 4096^3 5 809 -> 4 880, 8192^3 5 980 -> 4 600 (a six-fold K extent: 5 857, 5 776); on the other side of the
// line 8 x 1024^3 109 -> 112 (128 tiles), 8192 x 3072 x 768 186 -> 212, 8192 x 50264 x 768 2 849 -> 2 905 (nothing runs under the end of a tile).
static bool f3_wide(const GemmDesc& g) {
  const int64_t tiles = (g.m + 2 * kF3Bm - 1) / (2 * kF3Bm) * ((g.n + kFwBn - 1) / kFwBn) * g.batch;
  return g.k >= 1024 && tiles >= 3 * (sm_count() / 2);
}

// float32 A [m, k] with rows along k; B [k, n] with either dimension along its rows; bytes of the workspace for the planes and shares
bool f32x3_eligible(const GemmDesc& g) {
  if (g.dtype != DType::F32 || g.b_dtype != DType::F32 || g.batch_inner != 1 || g.k % 8 || g.a_col != 1 || g.a_row % 4 || g.a_batch % 4 || g.b_batch % 4) return false;
  if (g.ep.b_scales || g.ep.argmax_keys || g.ep.ln_stats || g.ep.stats_out || g.ep.stats_zero || g.ep.glu_n || g.ln_gamma) return false;
  if (g.m > 0x3fffffff || g.n > 0x3fffffff || g.k > 0x3fffffff || g.batch > 65535) return false;
  if (g.b_col == 1) { if (g.n % 8 || g.b_row % 4) return false; }
  else if (g.b_row != 1 || g.b_col % 4) return false;
  return aligned16(g.a) && aligned16(g.b);
}
static int64_t f3_pad(int64_t bytes) { return (bytes + 255) / 256 * 256; }
int64_t f32x3_workspace(const GemmDesc& g) {
  const int64_t ca = g.batch > 1 && g.a_batch ? g.batch : 1, cb = g.batch > 1 && g.b_batch ? g.batch : 1;
  const int s = f3_wide(g) ? 1 : f32x3_splits(g.m, g.n, g.k, g.batch);
  return 256 + f3_pad(6 * ca * g.m * g.k) + f3_pad(6 * cb * g.n * g.k) + (s > 1 ? (int64_t)s * g.batch * g.m * ((g.n + 3) / 4 * 4) * 4 : 0);
}

Status matmul_f32x3(cudaStream_t s, const GemmDesc& g, void* workspace) {
  if (!f32x3_eligible(g) || !workspace || !aligned16(workspace)) return Status::invalid("matmul_f32x3: operands");
  int* st = matmul_status_word();
  if (!st) return Status::compute("matmul: the kernel workspace is not initialised");
  const int64_t ca = g.batch > 1 && g.a_batch ? g.batch : 1, cb = g.batch > 1 && g.b_batch ? g.batch : 1;
  const bool b_mn = g.b_col == 1, wide = f3_wide(g);
  uint8_t* ws = static_cast<uint8_t*>(workspace) + 256;     // in front: the call whose operands hold a finite number beyond bf16
  static std::atomic<unsigned long long> calls{0x9e3779b97f4a7c15ull};      // what a pooled buffer holds is hardly ever the next call's (it would cost time only)
  unsigned long long* note = static_cast<unsigned long long*>(workspace);
  const unsigned long long call = calls.fetch_add(1, std::memory_order_relaxed);
  __nv_bfloat16* pa = reinterpret_cast<__nv_bfloat16*>(ws);
  __nv_bfloat16* pb = reinterpret_cast<__nv_bfloat16*>(ws + f3_pad(6 * ca * g.m * g.k));
  const int64_t b_rows = b_mn ? g.k : g.n, b_cols = b_mn ? g.n : g.k;
  PlaneJob ja{static_cast<const float*>(g.a), pa, g.m, g.k, g.a_row, g.a_batch, (int)ca, grid_for(ca * g.m * (g.k / 8), 256, 4)};
  PlaneJob jb{static_cast<const float*>(g.b), pb, b_rows, b_cols, b_mn ? g.b_row : g.b_col, g.b_batch, (int)cb, grid_for(cb * b_rows * (b_cols / 8), 256, 8)};
  cudaError_t e = launch_pdl(f32_planes_kernel, dim3((unsigned)(ja.blocks + jb.blocks)), dim3(256), 0, s, ja, jb, note, call);
  if (e != cudaSuccess) return cuda_status(e, "matmul_f32x3 planes");
  CUtensorMap ma, mb;
  AG_RETURN_IF_ERROR(make_map(&ma, DType::BF16, pa, (uint64_t)g.k, (uint64_t)g.m, 3, (uint64_t)ca, (uint64_t)g.k, (uint64_t)(g.m * g.k), (uint64_t)(3 * g.m * g.k), kF3Bk, kF3Bm));
  AG_RETURN_IF_ERROR(make_map(&mb, DType::BF16, pb, (uint64_t)b_cols, (uint64_t)b_rows, 3, (uint64_t)cb, (uint64_t)b_cols, (uint64_t)(b_rows * b_cols), (uint64_t)(3 * b_rows * b_cols), 64, 64));
  F3Params p;
  p.c = static_cast<float*>(g.c); p.bias = static_cast<const float*>(g.ep.bias); p.residual = static_cast<const float*>(g.ep.residual);
  p.alpha = g.ep.alpha; p.act = (int)g.ep.act; p.m = (int)g.m; p.n = (int)g.n; p.batch = (int)g.batch; p.a_one = ca == 1; p.b_one = cb == 1;
  p.num_kb = (int)((g.k + kF3Bk - 1) / kF3Bk); p.tiles_m = (int)((g.m + 2 * kF3Bm - 1) / (2 * kF3Bm)); p.tiles_n = (int)((g.n + (wide ? kFwBn : kF3Bn) - 1) / (wide ? kFwBn : kF3Bn));
  p.splits = wide ? 1 : f32x3_splits(g.m, g.n, g.k, g.batch); p.kb_per_split = (p.num_kb + p.splits - 1) / p.splits;
  p.c_row = g.c_row; p.c_batch = g.c_batch; p.p_row = (g.n + 3) / 4 * 4; p.status = st;
  p.a = static_cast<const float*>(g.a); p.b = static_cast<const float*>(g.b); p.k = (int)g.k; p.a_row = g.a_row; p.a_batch = g.a_batch; p.b_row = g.b_row; p.b_col = g.b_col; p.b_batch = g.b_batch;
  p.note = note; p.call = call;
  p.partial = p.splits > 1 ? reinterpret_cast<float*>(ws + f3_pad(6 * ca * g.m * g.k) + f3_pad(6 * cb * g.n * g.k)) : nullptr;
  p.vec = aligned16(g.c) && g.c_row % 4 == 0 && g.c_batch % 4 == 0 && (!g.ep.residual || aligned16(g.ep.residual)) ? 1 : 0;
  static bool attr = false;
  if (!attr) {
    e = cudaFuncSetAttribute(gemm_f32x3_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kF3Smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_f32x3_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kF3Smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_f32x3_wide_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_f32x3_wide_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwSmem);
    if (e != cudaSuccess) return cuda_status(e, "matmul_f32x3 smem attribute");
    attr = true;
  }
  const long long units = (long long)p.tiles_m * p.tiles_n * p.batch * p.splits;
  const dim3 grid((unsigned)(2 * std::min<long long>(units, sm_count() / 2)));
  if (wide)
    e = b_mn ? launch_pdl(gemm_f32x3_wide_kernel<true>, grid, dim3(kF3Threads), (size_t)kFwSmem, s, ma, mb, p) : launch_pdl(gemm_f32x3_wide_kernel<false>, grid, dim3(kF3Threads), (size_t)kFwSmem, s, ma, mb, p);
  else e = b_mn ? launch_pdl(gemm_f32x3_kernel<true>, grid, dim3(kF3Threads), (size_t)kF3Smem, s, ma, mb, p) : launch_pdl(gemm_f32x3_kernel<false>, grid, dim3(kF3Threads), (size_t)kF3Smem, s, ma, mb, p);
  if (e != cudaSuccess) return cuda_status(e, "matmul_f32x3");
  if (p.splits > 1) {
    e = launch_pdl(f32x3_finish_kernel, dim3((unsigned)grid_for((int64_t)p.batch * p.m * (p.p_row / 4), 256, 8)), dim3(256), 0, s, p);
    if (e != cudaSuccess) return cuda_status(e, "matmul_f32x3 shares");
  }
  return Status::OK();
}

}}  // namespace ag::k
