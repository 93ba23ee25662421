// Kernels of the parallel gated block: both sublayers read norms of the same residual row, the
// mixer's input is mixed with the previous token's (token shift), and each sublayer's result is
// scaled by a learned sigmoid gate before both are added to the residual stream.
//
//   n = x / sqrt(mean_g(x^2) + eps)        per group g of E / groups consecutive elements
//   a = n * w1,  b = n * w2                (one normalisation, two weight vectors)
//   m = a + (a_prev - a) * s               a_prev: the a of the request's previous token
//   x += y1 * sigmoid(g1 + c1) + (y2 + c2) * sigmoid(g2 + c3)
//
// Everything here is float32 arithmetic on the float32 residual stream; only a, m and b leave in
// the compute dtype, as inputs of the products that follow.  The previous token's a is found in
// the batch (the row before, recomputed from x with the same reduction tree, so that the value is
// bit-equal to what a step that ended on that token left behind) or, for the first token of a
// portion, in the request's state row.  A portion's last a goes to a staging row first and is
// copied into the state by the block's last kernel: the state is read and written by different
// launches, never by blocks of one grid.
#include <initializer_list>

#include "common.cuh"
#include "partials.cuh"

constexpr int GB_THREADS = 256;
constexpr int GB_MAX_GROUPS = 512;

// Four neighbouring values: loads of 16 bytes (zeros where there is no vector) and one store in the output type.
// The three kernels of a prompt portion move every element once and are bound by memory; with a 4-byte access per element
// and thread too few bytes were on their way (B200, 1,500 tokens x 2,048 / 5,632, us a launch within a step, before -> after:
// norm_pair_shift 21 -> 11, bias_glu 36 -> 21, gated_residual 36 -> 20).
template <typename T> __device__ __forceinline__ void gb_store4(T* p, float a, float b, float c, float d) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack2<T>(a, b), pack2<T>(c, d));
}
template <> __device__ __forceinline__ void gb_store4<float>(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ float4 gb_load4(const float* p, int i) { return *reinterpret_cast<const float4*>(p + i); }
__device__ __forceinline__ float4 gb_load4_or_zero(const float* p, int i) { return p ? gb_load4(p, i) : make_float4(0.f, 0.f, 0.f, 0.f); }
// Whether all of these (null ones aside) lie on 16-byte boundaries.
static bool gb_aligned(std::initializer_list<const void*> ps) {
  for (const void* p : ps)
    if ((uintptr_t)p & 15) return false;
  return true;
}

// 1 / sqrt(mean(part^2) + eps) of every group of row xr into inv[0 .. groups): warp w takes groups
// w, w + warps, ...; a lane walks its group with stride 32, then the lanes meet in a butterfly.
// The tree depends on (E, groups) alone.  Ends with a barrier.
__device__ __forceinline__ void group_inverse_rms(const float* __restrict__ xr, int E, int groups, float eps, float* inv) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int Eg = E / groups;
  for (int g = warp; g < groups; g += nw) {
    const float* p = xr + (size_t)g * Eg;
    float ss = 0.f;
    for (int i0 = lane; i0 < Eg; i0 += 32 * 8) {     // (eight loads on their way at a time; a zero changes no sum)
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = i0 + 32 * k < Eg ? p[i0 + 32 * k] : 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) ss = fmaf(v[k], v[k], ss);
    }
    ss = warp_sum(ss);
    if (lane == 0) inv[g] = 1.0f / sqrtf(ss / (float)Eg + eps);
  }
  __syncthreads();
}

// ---------------------------------------------------------------- embedding with scale and learned positions
template <typename T>
__global__ void embedding_scaled_kernel(const T* __restrict__ table, const int* __restrict__ ids, float* __restrict__ out, int E,
                                        int V, float scale, const T* __restrict__ pos_table, const int* __restrict__ positions,
                                        int n_pos, int* __restrict__ err) {
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x;
  const int id = ids[t];
  const bool ok = id >= 0 && id < V;
  if (!ok && threadIdx.x == 0) atomicExch(err, 1);
  const T* row = table + (size_t)(ok ? id : 0) * E;
  const T* prow = nullptr;
  if (pos_table != nullptr) {
    const int p = positions[t];
    if (p < 0 || p >= n_pos) {
      if (threadIdx.x == 0) atomicExch(err, 2);
    } else {
      prow = pos_table + (size_t)p * E;
    }
  }
  float* o = out + (size_t)t * E;
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    float v = ok ? to_f32<T>(row[i]) * scale : 0.f;
    if (prow != nullptr) v += to_f32<T>(prow[i]);
    o[i] = v;
  }
}

// out[t] = table[ids[t]] * scale (+ pos_table[positions[t]] when a position table is given), float32.
FERRUM_API int ferrum_embedding_scaled(const void* table, int dtype, const int* ids, float* out, int n_tokens, int E, int V,
                                       float scale, const void* pos_table, const int* positions, int n_pos, int* err_flag,
                                       cudaStream_t stream) {
  FERRUM_CHECK_ARG(n_tokens >= 0 && E > 0 && V > 0, "embedding: bad sizes T=%d E=%d V=%d", n_tokens, E, V);
  FERRUM_CHECK_ARG(pos_table == nullptr || (positions != nullptr && n_pos > 0), "embedding: positions missing");
  if (n_tokens == 0) return 0;
  const int threads = E >= 1024 ? 256 : 128;
  FERRUM_DISPATCH_DTYPE(dtype, T, launch_kernel(embedding_scaled_kernel<T>, n_tokens, threads, 0, stream, (const T*)table, ids, out, E, V,
                                                scale, (const T*)pos_table, positions, n_pos, err_flag));
  FERRUM_CHECK_LAUNCH("embedding_scaled");
  return 0;
}

// ---------------------------------------------------------------- grouped RMS norm (rows may be gathered)
template <typename TOut>
__global__ void __launch_bounds__(GB_THREADS)
group_norm_kernel(const float* __restrict__ x, const float* __restrict__ w, TOut* __restrict__ out, const int* __restrict__ rows, int E,
                  int groups, float eps) {
  __shared__ float inv[GB_MAX_GROUPS];
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x;
  const float* xr = x + (size_t)(rows ? rows[r] : r) * E;
  group_inverse_rms(xr, E, groups, eps, inv);
  const int Eg = E / groups;
  TOut* o = out + (size_t)r * E;
  for (int i = threadIdx.x; i < E; i += blockDim.x) o[i] = from_f32<TOut>(xr[i] * inv[i / Eg] * w[i]);
}

FERRUM_API int ferrum_group_norm(const float* x, const float* w, void* out, int out_dtype, const int* rows, int n_rows, int E,
                                 int groups, float eps, cudaStream_t stream) {
  FERRUM_CHECK_ARG(n_rows >= 0 && E > 0 && groups > 0 && groups <= GB_MAX_GROUPS && E % groups == 0,
                   "group norm: bad sizes rows=%d E=%d groups=%d", n_rows, E, groups);
  FERRUM_CHECK_ARG(eps > 0.f, "group norm: eps must be positive");
  if (n_rows == 0) return 0;
  FERRUM_DISPATCH_DTYPE(out_dtype, T, launch_kernel(group_norm_kernel<T>, n_rows, GB_THREADS, 0, stream, x, w, (T*)out, rows, E, groups, eps));
  FERRUM_CHECK_LAUNCH("group_norm");
  return 0;
}

// ---------------------------------------------------------------- both norms and the token shift
// One block per token.  a, m, b: [T, E] in the compute dtype (b and w2 may be null: a layer without
// a second sublayer).  shift null: m = a.  state: [slots, E] float32, the a of every request's last
// token; stage: [requests of the batch, E] float32, receives the a of every portion's last token.
// VEC: four elements a thread at a time (E / groups a multiple of 4, everything on 16-byte boundaries).
template <typename TOut, bool VEC>
__global__ void __launch_bounds__(GB_THREADS)
norm_pair_shift_kernel(const float* __restrict__ x, const float* __restrict__ w1, const float* __restrict__ w2,
                       const float* __restrict__ shift, TOut* __restrict__ a_out, TOut* __restrict__ m_out, TOut* __restrict__ b_out,
                       const int* __restrict__ positions, const int* __restrict__ req_of_token, const int* __restrict__ q_start,
                       const int* __restrict__ slots, const float* __restrict__ state, float* __restrict__ stage, int E, int groups,
                       float eps) {
  __shared__ float inv[GB_MAX_GROUPS], inv_prev[GB_MAX_GROUPS];
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x;
  const int r = req_of_token[t];
  const bool first = t == q_start[r], last = t == q_start[r + 1] - 1;
  const float* xr = x + (size_t)t * E;
  group_inverse_rms(xr, E, groups, eps, inv);
  // where the previous token's a comes from: 0 nowhere (position 0), 1 the row before, 2 the state
  int prev = 0;
  if (shift != nullptr && positions[t] > 0) prev = first ? 2 : 1;
  const float* xp = xr - E;
  if (prev == 1) group_inverse_rms(xp, E, groups, eps, inv_prev);
  const float* sp = prev == 2 ? state + (size_t)slots[r] * E : nullptr;
  const int Eg = E / groups;
  if constexpr (VEC) {
    for (int i = threadIdx.x * 4; i < E; i += GB_THREADS * 4) {
      const int g = i / Eg;
      const float4 xv = gb_load4(xr, i), wv = gb_load4(w1, i);
      const float4 pv = gb_load4_or_zero(prev == 1 ? xp : (prev == 2 ? sp : nullptr), i);
      const float4 sv = gb_load4_or_zero(shift, i), w2v = gb_load4_or_zero(w2, i);
      const float xs[4] = {xv.x, xv.y, xv.z, xv.w}, ws[4] = {wv.x, wv.y, wv.z, wv.w}, ps[4] = {pv.x, pv.y, pv.z, pv.w};
      const float ss[4] = {sv.x, sv.y, sv.z, sv.w}, w2s[4] = {w2v.x, w2v.y, w2v.z, w2v.w};
      const float in = inv[g], ip = prev == 1 ? inv_prev[g] : 0.f;
      float a[4], m[4], b[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float n = xs[k] * in;
        a[k] = n * ws[k];
        m[k] = a[k];
        if (shift != nullptr) {
          const float ap = prev == 1 ? ps[k] * ip * ws[k] : ps[k];
          m[k] = a[k] + (ap - a[k]) * ss[k];
        }
        b[k] = n * w2s[k];
      }
      const size_t o = (size_t)t * E + i;
      gb_store4<TOut>(a_out + o, a[0], a[1], a[2], a[3]);
      gb_store4<TOut>(m_out + o, m[0], m[1], m[2], m[3]);
      if (b_out != nullptr) gb_store4<TOut>(b_out + o, b[0], b[1], b[2], b[3]);
      if (last && stage != nullptr) gb_store4<float>(stage + (size_t)r * E + i, a[0], a[1], a[2], a[3]);
    }
  } else
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    const int g = i / Eg;
    const float n = xr[i] * inv[g];
    const float a = n * w1[i];
    float m = a;
    if (shift != nullptr) {
      float ap = 0.f;
      if (prev == 1) ap = xp[i] * inv_prev[g] * w1[i];
      else if (prev == 2) ap = sp[i];
      m = a + (ap - a) * shift[i];
    }
    a_out[(size_t)t * E + i] = from_f32<TOut>(a);
    m_out[(size_t)t * E + i] = from_f32<TOut>(m);
    if (b_out != nullptr) b_out[(size_t)t * E + i] = from_f32<TOut>(n * w2[i]);
    if (last && stage != nullptr) stage[(size_t)r * E + i] = a;
  }
}

FERRUM_API int ferrum_norm_pair_shift(const float* x, const float* w1, const float* w2, const float* shift, void* a_out, void* m_out,
                                      void* b_out, int out_dtype, int n_tokens, const int* positions, const int* req_of_token,
                                      const int* q_start, const int* slots, const float* state, float* stage, int E, int groups,
                                      float eps, cudaStream_t stream) {
  FERRUM_CHECK_ARG(n_tokens >= 0 && E > 0 && groups > 0 && groups <= GB_MAX_GROUPS && E % groups == 0,
                   "norm pair: bad sizes T=%d E=%d groups=%d", n_tokens, E, groups);
  FERRUM_CHECK_ARG(eps > 0.f, "norm pair: eps must be positive");
  FERRUM_CHECK_ARG((b_out == nullptr) == (w2 == nullptr), "norm pair: second weight and second output go together");
  FERRUM_CHECK_ARG(shift == nullptr || (state != nullptr && stage != nullptr && slots != nullptr), "norm pair: a token shift needs its state");
  if (n_tokens == 0) return 0;
  const bool vec = E / groups % 4 == 0 && gb_aligned({x, w1, w2, shift, a_out, m_out, b_out, state, stage});
  FERRUM_DISPATCH_DTYPE(out_dtype, T, launch_kernel(vec ? norm_pair_shift_kernel<T, true> : norm_pair_shift_kernel<T, false>, n_tokens, GB_THREADS, 0,
                                                    stream, x, w1, w2, shift, (T*)a_out, (T*)m_out, (T*)b_out, positions, req_of_token, q_start,
                                                    slots, state, stage, E, groups, eps));
  FERRUM_CHECK_LAUNCH("norm_pair_shift");
  return 0;
}

// ---------------------------------------------------------------- biased gated linear unit
// act[t, f] = f(gu[t, f] + bg[f]) * (gu[t, F + f] + bu[f]); gu float32 rows of stride ld, act in the
// compute dtype.  kind 0: f = silu; 1: f = gelu with the tanh approximation; 2: the clamped unit of common.cuh
// made of both values and `limit`.  Biases may be null.
__device__ __forceinline__ float glu_act(float z, int kind) {
  if (kind == 0) return z / (1.0f + expf(-z));
  const float u = 0.7978845608028654f * (z + 0.044715f * z * z * z);
  return 0.5f * z * (1.0f + tanhf(u));
}
__device__ __forceinline__ float glu_of(float g, float u, int kind, float limit) {
  return kind == GLU_SWISH_CLAMP ? glu_swish_clamp(g, u, limit) : glu_act(g, kind) * u;
}

template <typename TOut>
__global__ void __launch_bounds__(256)
bias_glu_kernel(const float* __restrict__ gu, int ld, const float* __restrict__ bg, const float* __restrict__ bu, TOut* __restrict__ act,
                int ld_out, int F, int kind, float limit) {
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.y;
  const float* row = gu + (size_t)t * ld;
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < F; f += gridDim.x * blockDim.x) {
    const float g = row[f] + (bg ? bg[f] : 0.f), u = row[F + f] + (bu ? bu[f] : 0.f);
    act[(size_t)t * ld_out + f] = from_f32<TOut>(glu_of(g, u, kind, limit));
  }
}

// The same, four features a thread (F and both strides multiples of 4, 16-byte boundaries), from nine tokens on: with fewer the blocks are too
// few to gain from wide loads.  (B200, F = 5,632, us, one feature a thread / four: 1 token 1.09 / 1.22, 8 1.13 / 1.22, 16 1.31 / 1.30, 64 2.47 / 2.01, 1,500 35 / 17.)
constexpr int GLU_VEC_THREADS = 128, GLU_VEC_MIN_TOKENS = 9;
template <typename TOut>
__global__ void __launch_bounds__(GLU_VEC_THREADS)
bias_glu_vec_kernel(const float* __restrict__ gu, int ld, const float* __restrict__ bg, const float* __restrict__ bu, TOut* __restrict__ act,
                    int ld_out, int F, int kind, float limit) {
  pdl_launch();
  pdl_wait();
  const int f = (blockIdx.x * GLU_VEC_THREADS + threadIdx.x) * 4;
  if (f >= F) return;
  const float* row = gu + (size_t)blockIdx.y * ld;
  const float4 g = gb_load4(row, f), u = gb_load4(row + F, f), cg = gb_load4_or_zero(bg, f), cu = gb_load4_or_zero(bu, f);
  gb_store4<TOut>(act + (size_t)blockIdx.y * ld_out + f, glu_of(g.x + cg.x, u.x + cu.x, kind, limit), glu_of(g.y + cg.y, u.y + cu.y, kind, limit),
                  glu_of(g.z + cg.z, u.z + cu.z, kind, limit), glu_of(g.w + cg.w, u.w + cu.w, kind, limit));
}

FERRUM_API int ferrum_bias_glu(const float* gu, int ld, const float* bias_gate, const float* bias_up, void* act, int act_dtype,
                               int ld_out, int n_tokens, int F, int kind, float limit, cudaStream_t stream) {
  FERRUM_CHECK_ARG(n_tokens >= 0 && n_tokens <= 65535 * 32 && F > 0 && ld >= 2 * F && ld_out >= F, "bias glu: bad sizes T=%d F=%d", n_tokens, F);
  FERRUM_CHECK_ARG(kind >= 0 && kind <= GLU_SWISH_CLAMP, "bias glu: unknown activation %d", kind);
  if (n_tokens == 0) return 0;
  FERRUM_CHECK_ARG(n_tokens <= 65535, "bias glu: too many tokens");
  if (n_tokens >= GLU_VEC_MIN_TOKENS && F % 4 == 0 && ld % 4 == 0 && ld_out % 4 == 0 && gb_aligned({gu, bias_gate, bias_up, act})) {
    const dim3 vgrid((F / 4 + GLU_VEC_THREADS - 1) / GLU_VEC_THREADS, n_tokens);
    FERRUM_DISPATCH_DTYPE(act_dtype, T, launch_kernel(bias_glu_vec_kernel<T>, vgrid, dim3(GLU_VEC_THREADS), 0, stream, gu, ld, bias_gate, bias_up, (T*)act, ld_out, F, kind, limit));
    FERRUM_CHECK_LAUNCH("bias_glu");
    return 0;
  }
  const dim3 grid(min((F + 255) / 256, 64), n_tokens);
  FERRUM_DISPATCH_DTYPE(act_dtype, T, launch_kernel(bias_glu_kernel<T>, grid, dim3(256), 0, stream, gu, ld, bias_gate, bias_up, (T*)act, ld_out, F, kind, limit));
  FERRUM_CHECK_LAUNCH("bias_glu");
  return 0;
}

// The same from a product still in partials (deferred mode): one product of 2F + n_extra rows
// (gate | up | extra); the extra columns (another product of the same input) are summed into
// extra[t, :] (float32) on the way.
template <typename TOut>
__global__ void __launch_bounds__(256)
bias_glu_reduce_kernel(const float* __restrict__ bg, const float* __restrict__ bu, TOut* __restrict__ act, int ld_out, int F, int kind, float limit,
                       float* __restrict__ extra, int n_extra, const PartialLayout L) {
  __shared__ PartialTable tab;
  build_partial_table(L, tab);
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.y;
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < F + n_extra; f += gridDim.x * blockDim.x) {
    if (f < F) {
      const float g = partial_sum(L, tab, t, f) + (bg ? bg[f] : 0.f), u = partial_sum(L, tab, t, F + f) + (bu ? bu[f] : 0.f);
      act[(size_t)t * ld_out + f] = from_f32<TOut>(glu_of(g, u, kind, limit));
    } else {
      extra[(size_t)t * n_extra + (f - F)] = partial_sum(L, tab, t, 2 * F + (f - F));
    }
  }
}

FERRUM_API int ferrum_bias_glu_reduce(const float* bias_gate, const float* bias_up, void* act, int act_dtype, int ld_out, int n_tokens,
                                      int F, int kind, float limit, float* extra, int n_extra, const float* partials, const int* layout,
                                      cudaStream_t stream) {
  FERRUM_CHECK_ARG(n_tokens >= 0 && n_tokens <= 65535 && F > 0 && ld_out >= F && n_extra >= 0, "bias glu: bad sizes T=%d F=%d", n_tokens, F);
  FERRUM_CHECK_ARG(kind >= 0 && kind <= GLU_SWISH_CLAMP, "bias glu: unknown activation %d", kind);
  FERRUM_CHECK_ARG(n_extra == 0 || extra != nullptr, "bias glu: the extra columns need a place");
  if (n_tokens == 0) return 0;
  PartialLayout L;
  if (int r = partial_make_layout(partials, layout, &L)) return r;
  FERRUM_CHECK_ARG(2 * F + n_extra <= L.tiles * 128 && n_tokens <= L.acc_cols, "bias glu: the partials do not cover the rows");
  const dim3 grid(min((F + n_extra + 255) / 256, 64), n_tokens);
  FERRUM_DISPATCH_DTYPE(act_dtype, T, launch_kernel(bias_glu_reduce_kernel<T>, grid, dim3(256), 0, stream, bias_gate, bias_up, (T*)act, ld_out, F,
                                                    kind, limit, extra, n_extra, L));
  FERRUM_CHECK_LAUNCH("bias_glu_reduce");
  return 0;
}

// ---------------------------------------------------------------- gated residual sum
// x[t, i] += y1[t, i] * sigmoid(g1[t, i] + c1[i]) + (y2[t, i] + c2[i]) * sigmoid(g2[t, i] + c3[i]); the second term is
// left out when y2 is null.  All float32; every operand has its own row stride.  y1 and y2 may each be a
// product still in partials (deferred mode), summed while it is read.  The block of a
// portion's last token also copies the staged row of its request into the state.
__device__ __forceinline__ float gb_sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }
// One element of it.  Which products are fused into sums is written out: left to the compiler, the two kernels below
// rounded differently, and a token's bits depended on how many others were in the step.
__device__ __forceinline__ float gb_residual(float x, float v1, float z1, bool second, float v2, float z2) {
  float add = __fmul_rn(v1, gb_sigmoid(z1));
  if (second) add = __fmaf_rn(v2, gb_sigmoid(z2), add);
  return __fadd_rn(x, add);
}

__global__ void __launch_bounds__(GB_THREADS)
gated_residual_kernel(float* __restrict__ x, int E, const float* __restrict__ y1, int ld_y1, const float* __restrict__ g1, int ld_g1,
                      const float* __restrict__ c1, const float* __restrict__ y2, int ld_y2, const float* __restrict__ c2,
                      const float* __restrict__ g2, int ld_g2, const float* __restrict__ c3, const int* __restrict__ req_of_token,
                      const int* __restrict__ q_start, const int* __restrict__ slots, const float* __restrict__ stage,
                      float* __restrict__ state, const PartialLayout L1, const PartialLayout L2) {
  __shared__ PartialTable tab1, tab2;
  if (L1.ws != nullptr) build_partial_table(L1, tab1);
  if (L2.ws != nullptr) build_partial_table(L2, tab2);
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x;
  float* xr = x + (size_t)t * E;
  const bool second = y2 != nullptr || L2.ws != nullptr;
  // (with few tokens a row is shared out between gridDim.y blocks: summing partials is several loads per element)
  const int per = (E + gridDim.y - 1) / gridDim.y;
  const int lo = blockIdx.y * per, hi = min(E, lo + per);
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const float v1 = L1.ws != nullptr ? partial_sum(L1, tab1, t, i) : y1[(size_t)t * ld_y1 + i];
    float v2 = 0.f, z2 = 0.f;
    if (second) {
      v2 = (L2.ws != nullptr ? partial_sum(L2, tab2, t, i) : y2[(size_t)t * ld_y2 + i]) + (c2 ? c2[i] : 0.f);
      z2 = g2[(size_t)t * ld_g2 + i] + (c3 ? c3[i] : 0.f);
    }
    xr[i] = gb_residual(xr[i], v1, g1[(size_t)t * ld_g1 + i] + (c1 ? c1[i] : 0.f), second, v2, z2);
  }
  if (state != nullptr) {
    const int r = req_of_token[t];
    if (t == q_start[r + 1] - 1) {
      float* dst = state + (size_t)slots[r] * E;
      const float* src = stage + (size_t)r * E;
      for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) dst[i] = src[i];
    }
  }
}

// The same over whole rows, four elements a thread (no partials; E and the strides multiples of 4, 16-byte boundaries).
__global__ void __launch_bounds__(GB_THREADS)
gated_residual_vec_kernel(float* __restrict__ x, int E, const float* __restrict__ y1, int ld_y1, const float* __restrict__ g1, int ld_g1,
                          const float* __restrict__ c1, const float* __restrict__ y2, int ld_y2, const float* __restrict__ c2,
                          const float* __restrict__ g2, int ld_g2, const float* __restrict__ c3, const int* __restrict__ req_of_token,
                          const int* __restrict__ q_start, const int* __restrict__ slots, const float* __restrict__ stage,
                          float* __restrict__ state) {
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x;
  float* xr = x + (size_t)t * E;
  const float *y1r = y1 + (size_t)t * ld_y1, *g1r = g1 + (size_t)t * ld_g1;
  const float *y2r = y2 ? y2 + (size_t)t * ld_y2 : nullptr, *g2r = y2 ? g2 + (size_t)t * ld_g2 : nullptr;
#pragma unroll 2
  for (int i = threadIdx.x * 4; i < E; i += GB_THREADS * 4) {
    const float4 xv = gb_load4(xr, i), v1 = gb_load4(y1r, i), z1 = gb_load4(g1r, i), b1 = gb_load4_or_zero(c1, i);
    const float4 v2 = gb_load4_or_zero(y2r, i), z2 = gb_load4_or_zero(g2r, i), b2 = gb_load4_or_zero(c2, i), b3 = gb_load4_or_zero(c3, i);
    const float xs[4] = {xv.x, xv.y, xv.z, xv.w}, v1s[4] = {v1.x, v1.y, v1.z, v1.w}, z1s[4] = {z1.x, z1.y, z1.z, z1.w};
    const float b1s[4] = {b1.x, b1.y, b1.z, b1.w}, v2s[4] = {v2.x, v2.y, v2.z, v2.w}, z2s[4] = {z2.x, z2.y, z2.z, z2.w};
    const float b2s[4] = {b2.x, b2.y, b2.z, b2.w}, b3s[4] = {b3.x, b3.y, b3.z, b3.w};
    float o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = gb_residual(xs[k], v1s[k], z1s[k] + b1s[k], y2r != nullptr, v2s[k] + b2s[k], z2s[k] + b3s[k]);
    gb_store4<float>(xr + i, o[0], o[1], o[2], o[3]);
  }
  if (state != nullptr) {
    const int r = req_of_token[t];
    if (t == q_start[r + 1] - 1) {
      float* dst = state + (size_t)slots[r] * E;
      const float* src = stage + (size_t)r * E;
      for (int i = threadIdx.x * 4; i < E; i += GB_THREADS * 4) *reinterpret_cast<float4*>(dst + i) = gb_load4(src, i);
    }
  }
}

FERRUM_API int ferrum_gated_residual(float* x, int n_tokens, int E, const float* y1, int ld_y1, const float* g1, int ld_g1,
                                     const float* c1, const float* y2, int ld_y2, const float* c2, const float* g2, int ld_g2,
                                     const float* c3, const int* req_of_token, const int* q_start, const int* slots,
                                     const float* stage, float* state, const float* partials1, const int* layout1,
                                     const float* partials2, const int* layout2, cudaStream_t stream) {
  FERRUM_CHECK_ARG(n_tokens >= 0 && E > 0 && (y1 != nullptr || partials1 != nullptr) && g1 != nullptr, "gated residual: bad arguments");
  FERRUM_CHECK_ARG((y2 == nullptr && partials2 == nullptr) || g2 != nullptr, "gated residual: the second term needs its gate");
  PartialLayout L1{nullptr, 0, 0, 0, 0}, L2{nullptr, 0, 0, 0, 0};
  if (partials1 != nullptr) {
    if (int r = partial_make_layout(partials1, layout1, &L1)) return r;
    FERRUM_CHECK_ARG(E <= L1.tiles * 128 && n_tokens <= L1.acc_cols, "gated residual: the partials do not cover the rows");
  }
  if (partials2 != nullptr) {
    if (int r = partial_make_layout(partials2, layout2, &L2)) return r;
    FERRUM_CHECK_ARG(E <= L2.tiles * 128 && n_tokens <= L2.acc_cols, "gated residual: the partials do not cover the rows");
  }
  FERRUM_CHECK_ARG(state == nullptr || (stage != nullptr && slots != nullptr && q_start != nullptr && req_of_token != nullptr),
                   "gated residual: the state copy needs the batch description");
  if (n_tokens == 0) return 0;
  if (n_tokens > 64 && L1.ws == nullptr && L2.ws == nullptr && (E | ld_y1 | ld_g1 | (y2 ? ld_y2 | ld_g2 : 0)) % 4 == 0 &&
      gb_aligned({x, y1, g1, c1, y2, c2, y2 ? g2 : nullptr, c3, stage, state})) {
    launch_kernel(gated_residual_vec_kernel, dim3(n_tokens), dim3(GB_THREADS), 0, stream, x, E, y1, ld_y1, g1, ld_g1, c1, y2, ld_y2, c2, g2, ld_g2, c3,
                  req_of_token, q_start, slots, stage, state);
    FERRUM_CHECK_LAUNCH("gated_residual");
    return 0;
  }
  const int slices = n_tokens <= 64 ? max(1, min(16, E / 256)) : 1;
  launch_kernel(gated_residual_kernel, dim3(n_tokens, slices), dim3(GB_THREADS), 0, stream, x, E, y1, ld_y1, g1, ld_g1, c1, y2, ld_y2, c2, g2, ld_g2, c3,
                req_of_token, q_start, slots, stage, state, L1, L2);
  FERRUM_CHECK_LAUNCH("gated_residual");
  return 0;
}
