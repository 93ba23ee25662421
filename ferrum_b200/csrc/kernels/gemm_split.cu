// out[t, n] (=, +=) sum_k x[t, k] * w[n, k] for float32 operands on the tcgen05 tensor cores.
//
// The tensor cores have no float32 input type, but a float32 is exactly the sum of three bfloat16 values:
// h = v rounded to bfloat16, m = v - h rounded, l = v - h - m (both differences are exact, and l has at most seven
// bits left).  Of the nine products of two such sums six are formed, hh, hm, mh, mm, hl and lh; what is left out (ml, lm,
// ll) is below 2^-24 of a product of the two values, 3.5e-9 of it on average, and of either sign (parts that are cut off instead of
// rounded all have the value's sign: what is left out is then up to 2^-21, 4e-8 on average, and always makes the product smaller).
// bfloat16's exponents end where float32's do, so the low part of a value below some 2^-102 would be cut off: the parts are
// those of 2^24 v, which are zero or normal for every v, subnormal ones too, and an output is 2^-48 of its sum.  (Values from 2^103 and
// sums from 2^80 on overflow there; see the last paragraph.)
// A product of two bfloat16 values is exact in float32; what a sum loses, it loses when
// it is added up.  The matrix unit cuts off where it adds, so its accumulator is never the whole sum: it takes
// 64 elements of K at a time, the small terms first (24 instructions, of which only the last four add at
// full size), and the epilogue's warps add each such piece to the sum of the pieces before it in registers,
// rounded to nearest.  (Error of 300 rows of standard normal elements against float64, 2-norm over 2-norm: K = 3,072
// 1.1e-7, K = 8,192 1.2e-7; the CUDA cores' tiled kernel, one FFMA accumulator over K, 9.9e-7 and 1.6e-6.)
//
// The order of an output's sum is a function of N and K alone: pieces of 64 in K order within a range of K, and the
// ranges (their number depends on N and K) in K order.  A token's result does not depend on the other tokens.
//
// What bounds it: six bfloat16 products for one float32 product, so a sixth of the tensor cores' rate, some 270
// TFLOP/s against the 74 of the FFMA pipes' peak.  To keep the matrix unit fed, the weights are taken apart once
// per tile by four warps while they are in the pipeline: TMA brings 128 rows x 64 float32, a thread owns
// a row, and the three parts go to tensor memory, from where the matrix unit takes its A operand (no
// shared memory is written, and none is needed for the 48 KB of parts).  The tokens are taken apart by a kernel
// ahead of this one, once for all tiles of features (`split_rows_kernel`: 6 bytes an element, written to the L2).
// A tile is 128 features x up to 128 tokens: per piece of K 24 instructions of 64 clocks against about 600
// issue slots of conversion and summing in every scheduler.  Ranges of K are written to the workspace and added by
// `split_sum_kernel`: the last CTA of a tile adding them itself was a serial tail of some 25 us.
// Measured on a B200, us, FFMA tiles -> this: 300 tokens x [5120, 3072] 332 -> 70, x [3072, 3072] 332 -> 47, x [16384, 3072]
// 898 -> 173, x [3072, 8192] 909 -> 92; 1,024 tokens x [16384, 3072] 2,090 -> 453 (228 TFLOP/s: 1.37 PFLOP/s of bfloat16
// products, 0.84 of the measured burst peak).
//
// Roles (320 threads): warp 0 = TMA producer, warp 1 = TMEM owner and MMA issuer, warps 2..5 = sums and
// epilogue, warps 6..9 = conversion of the weights.  Every wait is bounded; on a timeout the kernel raises the
// error flag, lets the copies in flight land, frees its tensor memory and returns.
//
// Infinities, NaN and overflow: the parts of an infinite value are not finite either, and inf * 0 among them may give NaN
// where the plain sum gives an infinity.  An output that is not finite is therefore summed again, plainly, of the values as
// they are, by a whole warp (`plain16`, `plain_quads`): NaN, an infinity or a finite sum, as the CUDA cores' kernel gives it.
// (Only where finite terms overflow beside an infinity of the other sign does the order of the terms decide between the two.)
// Cost, B200, 300 tokens, one token with a NaN / all: x [3072, 3072] 52 -> 160 / 286 us, x [16384, 3072] 183 -> 183 / 292; the FFMA tiles
// take 334 and 908 whatever the values.
#include <algorithm>

#include <cuda.h>

#include "common.cuh"
#include "ptx_sm100.cuh"

using namespace sm100;

namespace {

constexpr int GS_TILE_N = 128;              // features per tile
constexpr int GS_TILE_T = 128;              // tokens per tile at most
constexpr int GS_KC = 64;                   // elements of K that the matrix unit sums before the piece is taken out
constexpr int GS_RAW_BYTES = GS_TILE_N * GS_KC * 4;
constexpr int GS_RAW_STAGES = 4;
constexpr int GS_X_STAGES = 2;
constexpr int GS_X_STAGE_BYTES = 3 * GS_TILE_T * GS_KC * 2;
constexpr int GS_SMEM_BYTES = GS_RAW_STAGES * GS_RAW_BYTES + GS_X_STAGES * GS_X_STAGE_BYTES + 1024 + 256;
constexpr int GS_A_COL = 2 * GS_TILE_T;     // tensor-memory columns: two accumulators, then two sets of weight parts
constexpr int GS_A_COLS = 3 * GS_KC / 2;
constexpr int GS_MAX_SPLITS = 8;
constexpr float GS_UP = 16777216.f, GS_DOWN = 1.f / GS_UP / GS_UP;   // 2^24 for each operand, 2^-48 for a sum

struct SplitParams {
  const float* x;
  const float* w;
  float* out;
  float* partials;
  int* err;
  int M, N, K, ldx, ldw, ldo;
  int bt, tiles_n, tiles_t, splits;
  int add;                 // 1: out += product
};

__device__ __forceinline__ void gs_tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
      "%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// (the caller waits: tcgen05.wait::st)
__device__ __forceinline__ void gs_tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// Two float32 values of a pair rounded to bfloat16, the first in the low half.
__device__ __forceinline__ uint32_t round2(float2 v) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
  return r;
}
// v - (the two bfloat16 values of h), in one instruction for both: exact where h is v rounded.
__device__ __forceinline__ float2 minus2(float2 v, uint32_t h) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %6};\n\t"
      "fma.rn.f32x2 a, a, b, c;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(__uint_as_float(h << 16)), "f"(__uint_as_float(h & 0xffff0000u)), "f"(-1.f), "f"(v.x), "f"(v.y));
  return r;
}
// Two float32 values, times GS_UP, as the sums of three bfloat16 values each, packed pairwise.
__device__ __forceinline__ void split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
  float2 v;
  asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmul.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
      : "=f"(v.x), "=f"(v.y)
      : "f"(a), "f"(b), "f"(GS_UP));
  h = round2(v);
  v = minus2(v, h);
  m = round2(v);
  l = round2(minus2(v, m));
}

// x [M, K] float32 -> planes [3, M, K] bfloat16 (h, m, l of GS_UP x).  K a multiple of 8, rows 16-byte aligned.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ x, int M, int K, int ldx, uint16_t* __restrict__ planes) {
  pdl_launch();
  pdl_wait();
  const int per_row = K / 8;
  const size_t plane = (size_t)M * K;
  const long long n = (long long)M * per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_row), k = (int)(i - (long long)t * per_row) * 8;
    const float4 a = *reinterpret_cast<const float4*>(x + (size_t)t * ldx + k);
    const float4 b = *reinterpret_cast<const float4*>(x + (size_t)t * ldx + k + 4);
    uint4 h, m, l;
    split2(a.x, a.y, h.x, m.x, l.x);
    split2(a.z, a.w, h.y, m.y, l.y);
    split2(b.x, b.y, h.z, m.z, l.z);
    split2(b.z, b.w, h.w, m.w, l.w);
    uint16_t* o = planes + (size_t)t * K + k;
    *reinterpret_cast<uint4*>(o) = h;
    *reinterpret_cast<uint4*>(o + plane) = m;
    *reinterpret_cast<uint4*>(o + 2 * plane) = l;
  }
}

// The outputs that are not finite among feature n of tokens t .. t + 15, summed again plainly in K order, and the others' scale: a
// whole warp, a lane per feature.  The lanes share the tokens' elements; once every such sum is a NaN the rest cannot change it.
__device__ __noinline__ void plain16(const SplitParams& p, int t, int n, float (&v)[16]) {
  unsigned own = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) own |= (unsigned)(n < p.N && t + j < p.M && !isfinite(v[j])) << j;
  const unsigned rows = __reduce_or_sync(0xffffffffu, own);
  const float* xr = p.x + (size_t)t * p.ldx;
  const float* wr = p.w + (size_t)min(n, p.N - 1) * p.ldw;
  float sum[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) sum[j] = 0.f;
  for (int k = 0; k < p.K; k += 8) {
    const float4 a = *reinterpret_cast<const float4*>(wr + k), b = *reinterpret_cast<const float4*>(wr + k + 4);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (rows >> j & 1) {
        const float4 c = *reinterpret_cast<const float4*>(xr + (size_t)j * p.ldx + k), d = *reinterpret_cast<const float4*>(xr + (size_t)j * p.ldx + k + 4);
        sum[j] = fmaf(c.x, a.x, sum[j]);
        sum[j] = fmaf(c.y, a.y, sum[j]);
        sum[j] = fmaf(c.z, a.z, sum[j]);
        sum[j] = fmaf(c.w, a.w, sum[j]);
        sum[j] = fmaf(d.x, b.x, sum[j]);
        sum[j] = fmaf(d.y, b.y, sum[j]);
        sum[j] = fmaf(d.z, b.z, sum[j]);
        sum[j] = fmaf(d.w, b.w, sum[j]);
      }
    }
    if ((k & 56) == 0) {
      bool lost = true;
#pragma unroll
      for (int j = 0; j < 16; ++j) lost = lost && (!(own >> j & 1) || isnan(sum[j]));
      if (__all_sync(0xffffffffu, lost)) break;
    }
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = own >> j & 1 ? sum[j] : v[j] * GS_DOWN;
}

// A whole warp, feature n in every lane: tokens t .. t + count - 1 (at most 16) go to `out`, the loads first, so that they overlap.
__device__ __forceinline__ void finish16(const SplitParams& p, int t, int n, int count, float* v) {
  const bool mine = n < p.N;
  float* o = p.out + (size_t)t * p.ldo + n;
  bool fine = true;
#pragma unroll
  for (int j = 0; j < 16; ++j) fine = fine && (j >= count || isfinite(v[j]));
  if (__all_sync(0xffffffffu, fine || !mine)) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] *= GS_DOWN;
  } else {
    float copy[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) copy[j] = v[j];
    plain16(p, t, n, copy);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = copy[j];
  }
  if (!mine) return;
  float r[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) r[j] = p.add && j < count ? o[(size_t)j * p.ldo] : 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j)
    if (j < count) o[(size_t)j * p.ldo] = p.add ? r[j] + v[j] : v[j];
}

// Features n .. n + count - 1 of token t in every lane, at most four, of which the bits of `bad` are to be summed again (none: v is
// handed back): a whole warp takes one lane's quad after the other, lane l the elements 4 l .. 4 l + 3 of every 128, and the lanes' sums
// meet at the end.  (A thread on its own walked K in 7 ms where one token of a 3072 x 3072 product had a NaN.)
__device__ __noinline__ float4 plain_quads(const SplitParams& p, int t, int n, int count, unsigned bad, float4 v) {
  const int lane = threadIdx.x & 31;
  for (unsigned todo = __ballot_sync(0xffffffffu, bad != 0); todo; todo &= todo - 1) {
    const int from = __ffs(todo) - 1;
    const int ft = __shfl_sync(0xffffffffu, t, from), fn = __shfl_sync(0xffffffffu, n, from), fc = __shfl_sync(0xffffffffu, count, from);
    const unsigned fbad = __shfl_sync(0xffffffffu, bad, from);
    const float* xr = p.x + (size_t)ft * p.ldx;
    const float* wr = p.w + (size_t)fn * p.ldw;
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = 0; k0 < p.K; k0 += 256) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = k0 + u * 128 + lane * 4;
        if (k < p.K) {
          const float4 a = *reinterpret_cast<const float4*>(xr + k);
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            if (f < fc) {
              const float4 b = *reinterpret_cast<const float4*>(wr + (size_t)f * p.ldw + k);
              sum[f] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum[f]))));
            }
          }
        }
      }
      bool lost = true;      // a NaN in every sum that is asked for: the rest cannot change it
#pragma unroll
      for (int f = 0; f < 4; ++f) lost = lost && (!(fbad >> f & 1) || isnan(sum[f]));
      if (__any_sync(0xffffffffu, lost)) break;
    }
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) sum[f] += __shfl_xor_sync(0xffffffffu, sum[f], d);
    if (lane == from) v = make_float4(bad & 1 ? sum[0] : v.x, bad & 2 ? sum[1] : v.y, bad & 4 ? sum[2] : v.z, bad & 8 ? sum[3] : v.w);
  }
  return v;
}

// out[t, n] (=, +=) the sum of the ranges' partial sums, in K order; a thread takes four neighbouring features, and a warp
// stays together for the outputs that are summed again.
__global__ void __launch_bounds__(256)
split_sum_kernel(const SplitParams p) {
  pdl_launch();
  pdl_wait();
  const int lane = threadIdx.x & 31, groups = (p.N + 3) / 4;
  const size_t plane = (size_t)p.M * p.N;
  const long long quads = (long long)p.M * groups;
  const bool vec = p.N % 4 == 0 && p.ldo % 4 == 0 && ((uintptr_t)p.out & 15) == 0;
  for (long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < quads; i0 += (long long)gridDim.x * blockDim.x) {
    const long long i = min(i0 + lane, quads - 1);      // (lanes past the end go along with the last quad and write nothing)
    const int t = (int)(i / groups), n = (int)(i - (long long)t * groups) * 4, count = min(4, p.N - n);
    const bool mine = i0 + lane < quads;
    const float* src = p.partials + (size_t)t * p.N + n;
    float* o = p.out + (size_t)t * p.ldo + n;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), r = v;
    if (vec) {
      float4 part[GS_MAX_SPLITS];
#pragma unroll
      for (int q = 0; q < GS_MAX_SPLITS; ++q)
        if (q < p.splits) part[q] = __ldcg(reinterpret_cast<const float4*>(src + q * plane));
      if (p.add && mine) r = *reinterpret_cast<const float4*>(o);
      v = part[0];
#pragma unroll
      for (int q = 1; q < GS_MAX_SPLITS; ++q) {
        if (q < p.splits) {
          v.x += part[q].x;
          v.y += part[q].y;
          v.z += part[q].z;
          v.w += part[q].w;
        }
      }
    } else {
      for (int q = 0; q < p.splits; ++q) {
        v.x += __ldcg(src + q * plane);
        if (count > 1) v.y += __ldcg(src + q * plane + 1);
        if (count > 2) v.z += __ldcg(src + q * plane + 2);
        if (count > 3) v.w += __ldcg(src + q * plane + 3);
      }
      if (p.add && mine) {
        r.x = o[0];
        if (count > 1) r.y = o[1];
        if (count > 2) r.z = o[2];
        if (count > 3) r.w = o[3];
      }
    }
    const unsigned bad = !mine ? 0u : (unsigned)!isfinite(v.x) | (unsigned)!isfinite(v.y) << 1 | (unsigned)!isfinite(v.z) << 2 | (unsigned)!isfinite(v.w) << 3;
    v = make_float4(v.x * GS_DOWN, v.y * GS_DOWN, v.z * GS_DOWN, v.w * GS_DOWN);
    if (__any_sync(0xffffffffu, bad != 0)) v = plain_quads(p, t, n, count, bad, v);
    if (!mine) continue;
    if (p.add) v = make_float4(r.x + v.x, r.y + v.y, r.z + v.z, r.w + v.w);
    if (vec) {
      *reinterpret_cast<float4*>(o) = v;
      continue;
    }
    o[0] = v.x;
    if (count > 1) o[1] = v.y;
    if (count > 2) o[2] = v.z;
    if (count > 3) o[3] = v.w;
  }
}

__global__ void __launch_bounds__(320, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const SplitParams p) {
  extern __shared__ uint8_t gs_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)gs_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  __shared__ int ep_stop;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t raw_base = smem_u32(smem), x_base = raw_base + GS_RAW_STAGES * GS_RAW_BYTES;
  const uint32_t bar_base = x_base + GS_X_STAGES * GS_X_STAGE_BYTES;
  auto raw_full = [&](int s) { return bar_base + 8u * s; };
  auto raw_empty = [&](int s) { return bar_base + 8u * (GS_RAW_STAGES + s); };
  auto x_full = [&](int s) { return bar_base + 8u * (2 * GS_RAW_STAGES + s); };
  auto x_empty = [&](int s) { return bar_base + 8u * (2 * GS_RAW_STAGES + GS_X_STAGES + s); };
  constexpr int B2 = 2 * GS_RAW_STAGES + 2 * GS_X_STAGES;
  auto a_full = [&](int b) { return bar_base + 8u * (B2 + b); };
  auto a_empty = [&](int b) { return bar_base + 8u * (B2 + 2 + b); };
  auto acc_full = [&](int b) { return bar_base + 8u * (B2 + 4 + b); };
  auto acc_empty = [&](int b) { return bar_base + 8u * (B2 + 6 + b); };
  static_assert((B2 + 8) * 8 <= 256, "the barriers do not fit their place");

  if (threadIdx.x == 0) {
    abort_flag = 0;
    prefetch_tensormap(&tmap_w);
    prefetch_tensormap(&tmap_x);
    for (int s = 0; s < GS_RAW_STAGES; ++s) {
      mbar_init(raw_full(s), 1);
      mbar_init(raw_empty(s), 4);      // the four converting warps
    }
    for (int s = 0; s < GS_X_STAGES; ++s) {
      mbar_init(x_full(s), 1);
      mbar_init(x_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(a_full(b), 4);
      mbar_init(a_empty(b), 1);
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), 4);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;
  volatile int* abort_p = &abort_flag;
  const int nkb = (p.K + GS_KC - 1) / GS_KC;
  // An item is one range of K of one tile; the items of a tile of features follow each other, so that the
  // token tiles which read the same weights run at the same time.
  const int items = p.tiles_n * p.splits * p.tiles_t;
  auto item_of = [&](int item, int& n0, int& t0, int& seg) {
    const int r = item / p.tiles_t;
    t0 = (item - r * p.tiles_t) * p.bt;
    seg = r % p.splits;
    n0 = r / p.splits * GS_TILE_N;
  };
  auto first_kb = [&](int seg) { return (int)((long long)nkb * seg / p.splits); };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    // The weights run GS_LAG pieces ahead of the tokens: their ring is deeper, and they wait for no kernel.
    constexpr int GS_LAG = GS_RAW_STAGES - GS_X_STAGES;
    if (elect_one()) {
      const uint32_t x_plane = (uint32_t)p.bt * GS_KC * 2;
      int wi = blockIdx.x, xi = blockIdx.x;            // items of the two streams
      int wn0, wt0, wseg, xn0, xt0, xseg, wkb = 0, wend = 0, xkb = 0, xend = 0;
      if (wi < items) {
        item_of(wi, wn0, wt0, wseg);
        wkb = first_kb(wseg);
        wend = first_kb(wseg + 1);
        item_of(xi, xn0, xt0, xseg);
        xkb = wkb;
        xend = wend;
      }
      bool ok = true, waited = false;
      for (int i = 0; ok && xi < items; ++i) {
        if (wi < items) {                              // piece i of the weights
          const int s = i % GS_RAW_STAGES;
          if (!mbar_wait(raw_empty(s), ((i / GS_RAW_STAGES) & 1) ^ 1, abort_p)) { ok = false; break; }
          mbar_expect_tx(raw_full(s), GS_RAW_BYTES);
          tma_load_2d(raw_base + s * GS_RAW_BYTES, &tmap_w, raw_full(s), wkb * GS_KC, wn0);
          tma_load_2d(raw_base + s * GS_RAW_BYTES + GS_RAW_BYTES / 2, &tmap_w, raw_full(s), wkb * GS_KC + GS_KC / 2, wn0);
          if (++wkb == wend) {
            wi += gridDim.x;
            if (wi < items) {
              item_of(wi, wn0, wt0, wseg);
              wkb = first_kb(wseg);
              wend = first_kb(wseg + 1);
            }
          }
        }
        if (i < GS_LAG) continue;
        if (!waited) {                                 // the tokens' parts come from the kernel ahead
          pdl_wait();
          pdl_launch();
          waited = true;
        }
        const int j = i - GS_LAG, s = j % GS_X_STAGES;  // piece j of the tokens
        if (!mbar_wait(x_empty(s), ((j / GS_X_STAGES) & 1) ^ 1, abort_p)) { ok = false; break; }
        mbar_expect_tx(x_full(s), 3 * x_plane);
        for (int q = 0; q < 3; ++q)
          tma_load_2d(x_base + s * GS_X_STAGE_BYTES + q * x_plane, &tmap_x, x_full(s), xkb * GS_KC, q * p.M + xt0);
        if (++xkb == xend) {
          xi += gridDim.x;
          if (xi < items) {
            item_of(xi, xn0, xt0, xseg);
            xkb = first_kb(xseg);
            xend = first_kb(xseg + 1);
          }
        }
      }
      if (!ok) {
        abort_flag = 1;
        atomicExch(p.err, 10);
      }
      if (!waited) {
        pdl_wait();
        pdl_launch();
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_16bit(GS_TILE_N, p.bt, false);
      const uint32_t x_plane = (uint32_t)p.bt * GS_KC * 2 >> 4;       // in the descriptor's units of 16 bytes
      const uint64_t desc0 = umma_desc_k_sw128(x_base);
      int i = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        int n0, t0, seg;
        item_of(item, n0, t0, seg);
        const int count = first_kb(seg + 1) - first_kb(seg);
        for (int c = 0; c < count; ++c, ++i) {
          const int b = i & 1, s = i % GS_X_STAGES;
          if (!mbar_wait(acc_empty(b), ((i >> 1) & 1) ^ 1, abort_p)) { abort_flag = 1; atomicExch(p.err, 13); ok = false; break; }
          if (!mbar_wait(x_full(s), (i / GS_X_STAGES) & 1, abort_p) || !mbar_wait(a_full(b), (i >> 1) & 1, abort_p)) {
            abort_flag = 1;
            atomicExch(p.err, 11);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem_base + b * GS_TILE_T;
          const uint32_t a = tmem_base + GS_A_COL + b * GS_A_COLS;
          const uint64_t xs = desc0 + (uint64_t)(s * (GS_X_STAGE_BYTES >> 4));
          // parts (weights, tokens), the smallest products first: l h, h l, m m, m h, h m, h h
#pragma unroll
          for (int term = 0; term < 6; ++term) {
            constexpr int WP[6] = {2, 0, 1, 1, 0, 0}, XP[6] = {0, 2, 1, 0, 1, 0};
            const uint64_t b_desc = xs + XP[term] * x_plane;
            const uint32_t a_cols = a + WP[term] * (GS_KC / 2);
#pragma unroll
            for (int kk = 0; kk < GS_KC / 16; ++kk) {
              umma_bf16_ts(d, a_cols + kk * 8, b_desc + (uint64_t)(kk * 32 >> 4), idesc, term > 0 || kk > 0);
            }
          }
          umma_commit(x_empty(s));
          umma_commit(a_empty(b));
          umma_commit(acc_full(b));
        }
      }
    }
  } else if (warp < 6) {
    // ------------------------------------------------------------ sums and epilogue (warps 2..5)
    const int quarter = warp & 3;
    const int n_local = quarter * 32 + lane;
    const int ep_tid = threadIdx.x - 64;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    int i = 0;
    bool ok = true;
    pdl_wait();
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      int n0, t0, seg;
      item_of(item, n0, t0, seg);
      const int count = first_kb(seg + 1) - first_kb(seg);
      const int n = n0 + n_local, valid = min(p.bt, p.M - t0);
      float sum[GS_TILE_T];
#pragma unroll
      for (int j = 0; j < GS_TILE_T; ++j) sum[j] = 0.f;
      for (int c = 0; c < count; ++c, ++i) {
        const int b = i & 1;
        ok = mbar_wait(acc_full(b), (i >> 1) & 1, abort_p);
        if (!ok) {
          abort_flag = 1;
          atomicExch(p.err, 12);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c0 = 0; c0 < GS_TILE_T; c0 += 32) {
          if (c0 < valid) {
            float v[32];
            gs_tmem_ld32(lane_addr + b * GS_TILE_T + c0, v);
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[c0 + j] += v[j];
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(b));
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (ep_tid == 0) ep_stop = *abort_p;
      asm volatile("bar.sync 1, 128;" ::: "memory");      // the four warps agree on going on
      if (ep_stop) break;
      if (p.splits == 1) {
#pragma unroll
        for (int c0 = 0; c0 < GS_TILE_T; c0 += 16)
          if (c0 < valid) finish16(p, t0 + c0, n, min(16, valid - c0), &sum[c0]);
        continue;
      }
      // a range of K of the tile: to the workspace [range][token][feature], for split_sum_kernel
      if (n < p.N) {
        float* mine = p.partials + ((size_t)seg * p.M + t0) * p.N + n;
#pragma unroll
        for (int j = 0; j < GS_TILE_T; ++j)
          if (j < valid) __stcg(mine + (size_t)j * p.N, sum[j]);
      }
    }
    tc_fence_before();
  } else {
    // ------------------------------------------------------------ conversion of the weights (warps 6..9)
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + GS_A_COL;
    int i = 0;
    bool ok = true;
    for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
      int n0, t0, seg;
      item_of(item, n0, t0, seg);
      const int count = first_kb(seg + 1) - first_kb(seg);
      for (int c = 0; c < count; ++c, ++i) {
        const int s = i % GS_RAW_STAGES, b = i & 1;
        ok = mbar_wait(raw_full(s), (i / GS_RAW_STAGES) & 1, abort_p);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint8_t* src = smem + s * GS_RAW_BYTES + row * 128;
        const uint32_t dst = lane_addr + b * GS_A_COLS;
        float4 f[GS_KC / 4];
#pragma unroll
        for (int v = 0; v < GS_KC / 4; ++v)           // 16-byte piece v & 7 of the row's 128 bytes; the TMA's swizzle: piece ^ (row % 8)
          f[v] = *reinterpret_cast<const float4*>(src + (v >> 3) * (GS_RAW_BYTES / 2) + (((v & 7) ^ (row & 7)) << 4));
        ok = mbar_wait(a_empty(b), ((i >> 1) & 1) ^ 1, abort_p);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int q = 0; q < 4; ++q) {                 // 16 elements: 8 columns of each part
          uint32_t h[8], m[8], l[8];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            split2(f[q * 4 + v].x, f[q * 4 + v].y, h[2 * v], m[2 * v], l[2 * v]);
            split2(f[q * 4 + v].z, f[q * 4 + v].w, h[2 * v + 1], m[2 * v + 1], l[2 * v + 1]);
          }
          gs_tmem_st8(dst + q * 8, h);
          gs_tmem_st8(dst + GS_KC / 2 + q * 8, m);
          gs_tmem_st8(dst + GS_KC + q * 8, l);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(raw_empty(s));
          mbar_arrive(a_full(b));
        }
      }
    }
    if (!ok) {
      abort_flag = 1;
      atomicExch(p.err, 15);
    }
  }

  __syncthreads();
  if (abort_flag && threadIdx.x == 0) {
    // let TMA copies that were already issued land before the CTA's shared memory goes away
    const long long t0c = clock64();
    while (clock64() - t0c < 2000000LL) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A row-major matrix in boxes of box_rows x 128 bytes with the 128-byte swizzle; what lies outside reads as zero.
int gs_tensor_map(CUtensorMap* out, bool f32, const void* ptr, long long rows, long long cols, long long ld, int box_rows) {
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult qres;
  static const EncodeTiledFn fn = [&]() -> EncodeTiledFn {
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
      return (EncodeTiledFn)sym;
    return nullptr;
  }();
  FERRUM_CHECK_ARG(fn != nullptr, "gemm_split: the driver does not export cuTensorMapEncodeTiled");
  const int esize = f32 ? 4 : 2;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * esize};
  cuuint32_t box[2] = {(cuuint32_t)(128 / esize), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FERRUM_CHECK_ARG(r == CUDA_SUCCESS, "gemm_split: cuTensorMapEncodeTiled failed with code %d (rows=%lld cols=%lld ld=%lld)", (int)r, rows, cols, ld);
  return 0;
}

// Ranges of K: as many as let one token tile's items fill the GPU, of 512 elements or more.  A function of N and K alone.
int gs_splits(int N, int K) {
  const int tiles_n = (N + GS_TILE_N - 1) / GS_TILE_N;
  return std::max(1, std::min(std::min(GS_MAX_SPLITS, 148 / tiles_n), K / 512));
}
struct GsShape {
  int M, N, bt, tiles_n, tiles_t, splits;
  GsShape(int M_, int N_, int K) : M(M_), N(N_) {
    tiles_n = (N + GS_TILE_N - 1) / GS_TILE_N;
    tiles_t = (M + GS_TILE_T - 1) / GS_TILE_T;
    bt = ((M + tiles_t - 1) / tiles_t + 15) / 16 * 16;   // equal tiles, a multiple of the instruction's 16
    splits = gs_splits(N, K);
  }
  long long partial_floats() const { return splits == 1 ? 0 : (long long)splits * M * N; }
};

}  // namespace

// Scratch of a product: floats[0] for the tokens' parts (3 bfloat16 each), floats[1] for partial sums.
FERRUM_API void ferrum_gemm_split_workspace(int M, int N, int K, long long* floats) {
  const GsShape s(std::max(1, M), N, K);
  floats[0] = ((long long)M * K * 3 + 1) / 2;
  floats[1] = s.partial_floats();
}

FERRUM_API int ferrum_gemm_split(const float* x, const float* w, float* out, int M, int N, int K, int ldx, int ldw, int ldo, int add,
                                 float* parts, long long parts_floats, float* partials, long long partial_floats, int* err_flag,
                                 cudaStream_t stream) {
  FERRUM_CHECK_ARG(M >= 0 && N > 0 && K > 0, "gemm_split: bad sizes M=%d N=%d K=%d", M, N, K);
  FERRUM_CHECK_ARG(err_flag != nullptr, "gemm_split: the error flag is required");
  if (M == 0) return 0;
  FERRUM_CHECK_ARG(K % 8 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0,
                   "gemm_split: K=%d must be a multiple of 8 and the rows (strides %d, %d) must start on 16 bytes", K, ldx, ldw);
  FERRUM_CHECK_ARG(ldx >= K && ldw >= K && ldo >= N, "gemm_split: a row stride is shorter than its row");
  const GsShape s(M, N, K);
  long long need[2];
  ferrum_gemm_split_workspace(M, N, K, need);
  FERRUM_CHECK_ARG(parts && parts_floats >= need[0] && ((uintptr_t)parts & 15) == 0, "gemm_split: needs %lld floats for the parts, got %lld", need[0], parts_floats);
  FERRUM_CHECK_ARG(need[1] == 0 || (partials && partial_floats >= need[1]), "gemm_split: needs %lld floats for partial sums, got %lld", need[1], partial_floats);
  FERRUM_CHECK_ARG(((uintptr_t)partials & 15) == 0, "gemm_split: the partial sums must be 16-byte aligned");
  FERRUM_CHECK_ARG((long long)s.tiles_n * s.tiles_t * s.splits < (1LL << 30) && 3LL * M < (1LL << 31), "gemm_split: too many tiles");
  static bool configured = false;
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GS_SMEM_BYTES);
    FERRUM_CHECK_ARG(e == cudaSuccess, "gemm_split: cannot reserve %d bytes of shared memory: %s", GS_SMEM_BYTES, cudaGetErrorString(e));
    configured = true;
  }
  CUtensorMap mw, mx;
  if (int r = gs_tensor_map(&mw, true, w, N, K, ldw, GS_TILE_N)) return r;
  if (int r = gs_tensor_map(&mx, false, parts, 3LL * M, K, K, s.bt)) return r;
  const long long pieces = (long long)M * (K / 8);
  const int blocks = (int)std::min<long long>((pieces + 255) / 256, 8LL * ferrum_sm_count());
  launch_kernel(split_rows_kernel, dim3(blocks), dim3(256), 0, stream, x, M, K, ldx, (uint16_t*)parts);
  FERRUM_CHECK_LAUNCH("split_rows");
  SplitParams p{x, w, out, partials, err_flag, M, N, K, ldx, ldw, ldo, s.bt, s.tiles_n, s.tiles_t, s.splits, add};
  const int grid = std::min(ferrum_sm_count(), s.tiles_n * s.tiles_t * s.splits);
  launch_kernel(gemm_split_kernel, dim3(grid), dim3(320), GS_SMEM_BYTES, stream, mw, mx, p);
  FERRUM_CHECK_LAUNCH("gemm_split");
  if (s.splits > 1) {
    const long long quads = (long long)M * ((N + 3) / 4);
    launch_kernel(split_sum_kernel, dim3((int)std::min<long long>((quads + 255) / 256, 8LL * ferrum_sm_count())), dim3(256), 0, stream, p);
    FERRUM_CHECK_LAUNCH("split_sum");
  }
  return 0;
}
