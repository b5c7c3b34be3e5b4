// Kernels between the products of a layer whose sublayers read the residual stream itself and whose results are
// normed, and the kernels that prepare queries, keys and values from float32 projections.  All arithmetic is float32;
// T below is the compute dtype (of q, of the cache and of rows that enter a product).
//
//   round_rows_kernel          x (float32) -> compute dtype
//   norm_add_kernel            x += y / rms(y) * w  (y a sublayer's float32 result); optionally also x in the compute dtype
//   norm_add_norm_kernel       the same addition, and the rows of the norm after it: rounded(x / rms(x) * w2); without x:
//                              x = y / rms(y) * w
//   token_gate_kernel          gelu_tanh(a) * table[id]
//   embed_pairs_kernel         table[id] * scale + pairs[(previous * a + id * b) mod n] (a sequence's first token: row n);
//                              the sequence's last token is kept per slot
//   qk_prepare_kernel          per token, from rows [q | k | v | gates]: short causal convolution of q and k over time,
//                              RMS norm (over a whole projection, or per head with one shared weight), rotation of a
//                              prefix of every head, k and v (own, mixed with another layer's, or the keys before the
//                              norm) into the paged cache, the gates' logits passed on
//   latent_rotate_append_kernel  per token, from rows [q heads of D + R | latent C | shared key part R]: the latent
//                              under its RMS norm and the turned key part go into the cache row [c | k_r | 0], the
//                              queries leave with their last R values turned
//   rotate_rows_kernel         float32 rows in place: a prefix of every head turned by position
#include "rb_rotary.cuh"

namespace {

// one or two neighbouring values (two: the address is a multiple of two values)
template <typename T> __device__ __forceinline__ void rb_store_values(T* dst, const float* y, int n);
template <> __device__ __forceinline__ void rb_store_values<float>(float* dst, const float* y, int n) {
  if (n == 2) *reinterpret_cast<float2*>(dst) = make_float2(y[0], y[1]);
  else dst[0] = y[0];
}
template <> __device__ __forceinline__ void rb_store_values<__nv_bfloat16>(__nv_bfloat16* dst, const float* y, int n) {
  if (n == 2) *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(y[0], y[1]);
  else dst[0] = __float2bfloat16_rn(y[0]);
}

template <typename T>
__global__ void __launch_bounds__(256) round_rows_kernel(T* out, const float* x, int64_t n) {
  rb_pdl_launch_dependents();
  rb_pdl_wait();
  // four values a thread and turn where the addresses allow 16-byte loads, the rest value by value
  const bool vec = ((uintptr_t)x % 16 == 0) && ((uintptr_t)out % (4 * sizeof(T)) == 0);
  const int64_t n4 = vec ? n / 4 : 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 v = *reinterpret_cast<const float4*>(x + 4 * i);
    const float y[4] = {v.x, v.y, v.z, v.w};
    rb_store_values<T>(out + 4 * i, y, 2);
    rb_store_values<T>(out + 4 * i + 2, y + 2, 2);
  }
  for (int64_t i = 4 * n4 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = rb_from_float<T>(x[i]);
}

// A block per row.  VEC: a thread holds NV times four values of both rows in registers (blockDim.x * NV * 4 >= E), all asked for at
// once, the weights before the wait for the kernel before; else the rows go through memory, with NV 0 four values at a time.  1 row
// of 2,048 values took 3.0 us of a step with a load of y for its sum and one of everything after it, so 1.8.
template <typename T, bool VEC, int NV>
__global__ void __launch_bounds__(1024) norm_add_kernel(float* x, const float* y,
                                                        const float* w, float eps, int E,
                                                        T* rounded) {
  rb_pdl_launch_dependents();
  __shared__ float scratch[33];
  const int64_t row = blockIdx.x;
  const float* yr = y + row * E;
  float* xr = x + row * E;
  if constexpr (VEC) {
    float ww[NV][4], v[NV][4], o[NV][4];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
      if (e < E) rb_load4(w + e, ww[i]);
    }
    rb_pdl_wait();
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
#pragma unroll
      for (int k = 0; k < 4; ++k) v[i][k] = 0.f;
      if (e < E) { rb_load4(yr + e, v[i]); rb_load4(xr + e, o[i]); }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) ss = fmaf(v[i][k], v[i][k], ss);
    ss = rb_block_sum_once(ss, scratch);
    const float r = 1.0f / sqrtf(ss / (float)E + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
      if (e < E) {
#pragma unroll
        for (int k = 0; k < 4; ++k) o[i][k] += v[i][k] * r * ww[i][k];
        rb_store4(xr + e, o[i]);
        if (rounded != nullptr) rb_store4(rounded + row * E + e, o[i]);
      }
    }
    return;
  }
  rb_pdl_wait();
  float ss = 0.f;
  if (NV == 0) {
    for (int e = threadIdx.x * 4; e < E; e += blockDim.x * 4) {
      float v[4];
      rb_load4(yr + e, v);
      ss += v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3];
    }
    ss = rb_block_sum(ss, scratch);
    const float r = 1.0f / sqrtf(ss / (float)E + eps);
    for (int e = threadIdx.x * 4; e < E; e += blockDim.x * 4) {
      float v[4], ww[4], o[4];
      rb_load4(yr + e, v);
      rb_load4(w + e, ww);
      rb_load4(xr + e, o);
#pragma unroll
      for (int k = 0; k < 4; ++k) o[k] += v[k] * r * ww[k];
      rb_store4(xr + e, o);
      if (rounded != nullptr)
#pragma unroll
        for (int k = 0; k < 4; ++k) rounded[row * E + e + k] = rb_from_float<T>(o[k]);
    }
    return;
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) ss += yr[e] * yr[e];
  ss = rb_block_sum(ss, scratch);
  const float r = 1.0f / sqrtf(ss / (float)E + eps);
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const float o = xr[e] + yr[e] * r * w[e];
    xr[e] = o;
    if (rounded != nullptr) rounded[row * E + e] = rb_from_float<T>(o);
  }
}

// A block per row: x (+)= y / rms(y) * w, then h = x / rms(x) * w2.  VEC: a thread holds NV times four values of the row in
// registers (blockDim.x * NV * 4 >= E); else the row goes through memory, each thread its own values.
template <typename T, bool VEC, int NV, bool AHEAD>
__global__ void __launch_bounds__(1024) norm_add_norm_kernel(float* x, const float* y,
                                                             const float* w, float eps, int E, int fresh,
                                                             T* h, const float* w2, float eps2) {
  rb_pdl_launch_dependents();
  __shared__ float scratch[33], scratch2[32];
  const int64_t row = blockIdx.x;
  const float* yr = y + row * E;
  float* xr = x + row * E;
  T* hr = h + row * E;
  if (VEC) {
    // The weights do not depend on the kernel before this one; with AHEAD the second ones are asked for here too, without it after the
    // first sum.  Sixteen values a thread and both weights do not fit 64 registers, which a few rows do not feel and many do: rows
    // of 8,192 values, asked for ahead and not: 1 2.7, 2.9 us, 2,000 41.5, 38.3; of 16,384 2,000 92, 80.
    float ww[NV][4], ww2[AHEAD ? NV : 1][4], v[NV][4], o[NV][4];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
      if (e < E) rb_load4(w + e, ww[i]);
      if (AHEAD && e < E) rb_load4(w2 + e, ww2[i]);
    }
    rb_pdl_wait();
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
#pragma unroll
      for (int k = 0; k < 4; ++k) v[i][k] = o[i][k] = 0.f;
      if (e < E) {
        rb_load4(yr + e, v[i]);
        if (!fresh) rb_load4(xr + e, o[i]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) ss = fmaf(v[i][k], v[i][k], ss);
    }
    ss = rb_block_sum_once(ss, scratch);
    const float r = 1.0f / sqrtf(ss / (float)E + eps);
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
      if (e < E) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          o[i][k] += v[i][k] * r * ww[i][k];
          ss = fmaf(o[i][k], o[i][k], ss);
        }
        rb_store4(xr + e, o[i]);
        if (!AHEAD) rb_load4(w2 + e, ww[i]);
      }
    }
    ss = rb_block_sum_once(ss, scratch2);
    const float r2 = 1.0f / sqrtf(ss / (float)E + eps2);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int e = (i * blockDim.x + threadIdx.x) * 4;
      if (e < E) {
#pragma unroll
        for (int k = 0; k < 4; ++k) o[i][k] = o[i][k] * r2 * (AHEAD ? ww2[AHEAD ? i : 0][k] : ww[i][k]);
        rb_store4(hr + e, o[i]);
      }
    }
    return;
  }
  rb_pdl_wait();
  float ss = 0.f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) ss = fmaf(yr[e], yr[e], ss);
  ss = rb_block_sum(ss, scratch);
  const float r = 1.0f / sqrtf(ss / (float)E + eps);
  ss = 0.f;
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    const float o = (fresh ? 0.f : xr[e]) + yr[e] * r * w[e];
    xr[e] = o;
    ss = fmaf(o, o, ss);
  }
  ss = rb_block_sum(ss, scratch);
  const float r2 = 1.0f / sqrtf(ss / (float)E + eps2);
  for (int e = threadIdx.x; e < E; e += blockDim.x) hr[e] = rb_from_float<T>(xr[e] * r2 * w2[e]);
}

__device__ __forceinline__ float gelu_tanh_(float z) {
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

template <typename T, typename TT>
__global__ void __launch_bounds__(256) token_gate_kernel(T* out, const float* a, int64_t lda,
                                                         const TT* table, const int* ids,
                                                         int64_t n, int dim) {
  rb_pdl_launch_dependents();
  rb_pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / dim;
    const int j = (int)(i % dim);
    out[i] = rb_from_float<T>(gelu_tanh_(a[t * lda + j]) * rb_to_float<TT>(table[(int64_t)ids[t] * dim + j]));
  }
}

// A block per row.  add: the embedded rows are made; update: the run's last row leaves its token in `previous`.
// single: every row is a run of its own (a decode step; rows that pad a captured step may share a slot).  A step of
// runs of several rows takes two launches (add, then update), because a run's first row reads what its last row writes.
template <typename TT>
__global__ void __launch_bounds__(256) embed_pairs_kernel(float* out, const TT* table,
                                                          const TT* pairs, const int* ids,
                                                          const int* tok_pos, const int* tok_slot,
                                                          int* previous, int T, int E, int V, float scale,
                                                          int buckets, int mul_prev, int mul_cur, int add, int update,
                                                          int single) {
  rb_pdl_launch_dependents();
  rb_pdl_wait();
  const int t = blockIdx.x;
  const int slot = tok_slot[t], pos = tok_pos[t];
  int id = ids[t];
  id = id < 0 ? 0 : (id >= V ? V - 1 : id);
  const bool first = single || t == 0 || tok_slot[t - 1] != slot;
  const bool last = single || t == T - 1 || tok_slot[t + 1] != slot;
  if (add) {
    int row = buckets;
    if (pos > 0) {
      int prev = first ? previous[slot] : ids[t - 1];
      prev = prev < 0 ? 0 : (prev >= V ? V - 1 : prev);
      row = (int)(((int64_t)prev * mul_prev + (int64_t)id * mul_cur) % buckets);
    }
    const TT* a = table + (int64_t)id * E;
    const TT* b = pairs + (int64_t)row * E;
    for (int e = threadIdx.x; e < E; e += blockDim.x)
      out[(int64_t)t * E + e] = rb_to_float<TT>(a[e]) * scale + rb_to_float<TT>(b[e]);
  }
  if (update && last) {
    __syncthreads();                 // every thread of a single row's block has read the old value
    if (threadIdx.x == 0) previous[slot] = id;
  }
}

struct QkParams {
  const float* proj; int64_t ld;
  const float* conv_w; int K; float* tail; const int* tok_first;     // taps [C, K]; ring [n_slots, K, C]; null: rows are runs
  int norm_mode;                                                     // 0 none, 1 whole projection, 2 per head, one weight
  const float* q_norm_w; const float* k_norm_w; float eps;
  const double* freq; float magnitude; int rot_dim; int interleaved;
  const int* tok_pos; const int* tok_slot;
  int H, D, Dv;
  int values_are_keys;
  const float* mix_rows; int64_t mix_ld; float mix_weight;           // another layer's values of the same rows, or null
  int gate_heads;
  int staged;                                                        // the norms' weights wait in shared memory
};

// A block per token.  Shared memory: rot_dim sines and cosines, the C = (H + Kh) D convolved q and k values, a factor
// per head, the norms' weights.  Takes what qk_prepare_quads_kernel does not.
template <typename T>
__global__ void __launch_bounds__(1024) qk_prepare_kernel(T* q_out, T* gates_out, QkParams p,
                                                         RbPagedLayer cache) {
  rb_pdl_launch_dependents();
  __shared__ float scratch[33];
  extern __shared__ float s_mem[];
  const int H = p.H, D = p.D, Dv = p.Dv, Kh = cache.n_kv_heads, Dc = cache.head_dim;
  const int C = (H + Kh) * D;
  float* s_sincos = s_mem;
  float* s_qk = s_mem + p.rot_dim;
  float* s_fac = s_qk + C;
  float* s_nw = s_fac + H + Kh;                     // [q weights | k weights], of a head or of all
  const int t = blockIdx.x;
  const int pos = p.tok_pos[t], slot = p.tok_slot[t];
  const int64_t page0 = rb_page_offset(cache, slot, pos, 0), page_step = (int64_t)cache.page_size * Dc;      // kv head h: page0 + h * page_step
  const int nq = p.norm_mode == 1 ? H * D : (p.norm_mode == 2 ? D : 0), nk = p.norm_mode == 1 ? Kh * D : nq;
  if (p.staged)
    for (int i = threadIdx.x; i < nq + nk; i += blockDim.x) s_nw[i] = i < nq ? p.q_norm_w[i] : p.k_norm_w[i - nq];
  for (int i = threadIdx.x; i < p.rot_dim / 2; i += blockDim.x)
    angle_sincos(pos, p.freq[i], p.magnitude, &s_sincos[i], &s_sincos[p.rot_dim / 2 + i]);
  rb_pdl_wait();
  const float* row = p.proj + (int64_t)t * p.ld;
  if (p.conv_w != nullptr) {
    // tap by tap over all channels, so that a thread's loads of one pass do not wait for one another
    const int K = p.K;
    const int pos0 = p.tok_first != nullptr ? p.tok_pos[p.tok_first[t]] : pos;     // the run's first position
    for (int c = threadIdx.x; c < C; c += blockDim.x) s_qk[c] = p.conv_w[(int64_t)c * K + K - 1] * row[c];
    for (int back = 1; back < K && back <= pos; ++back) {
      const int at = pos - back;
      const float* src = at >= pos0 ? row - (int64_t)back * p.ld : p.tail + ((int64_t)slot * K + at % K) * C;
      for (int c = threadIdx.x; c < C; c += blockDim.x)
        s_qk[c] = fmaf(p.conv_w[(int64_t)c * K + K - 1 - back], src[c], s_qk[c]);
    }
    if (p.tok_first == nullptr && K > 1)                                           // a row that is its own run
      for (int c = threadIdx.x; c < C; c += blockDim.x) p.tail[((int64_t)slot * K + pos % K) * C + c] = row[c];
  } else {
    for (int c = threadIdx.x; c < C; c += blockDim.x) s_qk[c] = row[c];
  }
  __syncthreads();
  if (p.norm_mode == 1) {
    float ss = 0.f;
    for (int e = threadIdx.x; e < H * D; e += blockDim.x) ss += s_qk[e] * s_qk[e];
    ss = rb_block_sum(ss, scratch);
    const float rq = 1.0f / sqrtf(ss / (float)(H * D) + p.eps);
    ss = 0.f;
    for (int e = threadIdx.x; e < Kh * D; e += blockDim.x) ss += s_qk[H * D + e] * s_qk[H * D + e];
    ss = rb_block_sum(ss, scratch);
    const float rk = 1.0f / sqrtf(ss / (float)(Kh * D) + p.eps);
    for (int h = threadIdx.x; h < H + Kh; h += blockDim.x) s_fac[h] = h < H ? rq : rk;
  } else if (p.norm_mode == 2) {
    const int lane = threadIdx.x & 31;
    for (int h = threadIdx.x >> 5; h < H + Kh; h += blockDim.x >> 5) {
      float ss = 0.f;
      for (int e = lane; e < D; e += 32) ss += s_qk[h * D + e] * s_qk[h * D + e];
      ss = rb_warp_sum(ss);
      if (lane == 0) s_fac[h] = 1.0f / sqrtf(ss / (float)D + p.eps);
    }
  }
  __syncthreads();
  T* kdst = (T*)cache.k;
  T* vdst = (T*)cache.v;
  // a warp takes a head at a time (no division per value); a lane makes `step` neighbouring values of it at a time
  // (two where the cache rows have an even width)
  const int step = (Dc & 1) ? 1 : 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const int mode = p.norm_mode;
  for (int head = warp; head < H + Kh; head += n_warps) {
    const bool is_q = head < H;
    T* dst = is_q ? q_out + ((int64_t)t * H + head) * Dc : kdst + page0 + (head - H) * page_step;
    const float* src = s_qk + head * D;
    const float* nw = (p.staged ? s_nw + (is_q ? 0 : nq) : (is_q ? p.q_norm_w : p.k_norm_w)) + (mode == 1 ? (is_q ? head : head - H) * D : 0);
    const float fac = mode ? s_fac[head] : 1.f;
    auto val = [&](int i) { return mode ? src[i] * fac * nw[i] : src[i]; };
    for (int e0 = lane * step; e0 < Dc; e0 += 32 * step) {
      float y[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int e = e0 + k;
        y[k] = (k < step && e < D) ? turned(val, e, p.rot_dim, p.interleaved, s_sincos) : 0.f;
      }
      rb_store_values<T>(dst + e0, y, step);
    }
  }
  const int v_at = C;                                        // own values follow the keys in a row
  for (int kvh = warp; kvh < Kh; kvh += n_warps) {
    T* dst = vdst + page0 + kvh * page_step;
    const float* own = row + v_at + kvh * Dv;
    const float* other = p.mix_rows != nullptr ? p.mix_rows + (int64_t)t * p.mix_ld + kvh * Dv : nullptr;
    for (int e0 = lane * step; e0 < Dc; e0 += 32 * step) {
      float y[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int e = e0 + k;
        float v = 0.f;
        if (k < step && e < Dv) {
          if (p.values_are_keys) {
            v = s_qk[(H + kvh) * D + e];
          } else {
            v = own[e];
            if (other != nullptr) v = (1.0f - p.mix_weight) * v + p.mix_weight * other[e];
          }
        }
        y[k] = v;
      }
      rb_store_values<T>(dst + e0, y, step);
    }
  }
  if (p.gate_heads) {
    const int g_at = C + (p.values_are_keys ? 0 : Kh * Dv);
    for (int h = threadIdx.x; h < H; h += blockDim.x) gates_out[(int64_t)t * H + h] = rb_from_float<T>(row[g_at + h]);
  }
}

// The same in quads of neighbouring values: sizes and strides that are multiples of four, no convolution or one of four taps.
// A block per token, a chain of dependent reads in a step and, with many tokens, too little of the rows in flight, unless a thread asks
// for all of its share at once: taps, own row and the three before it (rows of the run, or of the ring before its start), the
// gates, the values, and only then makes anything of them.  Before the wait: positions, pages, weights, sines.  A warp takes a head,
// sums its squares (norm per head) and turns it, so that one barrier is all.  20 heads of 128 and 4 of values, of a whole request:
// a step's token 7.1 -> 5.2 us, 1,901 tokens with four taps 70 -> 31 us, without 36 -> 21 us.
template <typename T>
__global__ void __launch_bounds__(1024) qk_prepare_quads_kernel(T* q_out, T* gates_out, QkParams p, RbPagedLayer cache) {
  rb_pdl_launch_dependents();
  __shared__ float s_sum[2][32];
  extern __shared__ __align__(16) float s_mem[];
  const int H = p.H, D = p.D, Dv = p.Dv, Kh = cache.n_kv_heads, Dc = cache.head_dim;
  const int C = (H + Kh) * D, rhalf = p.rot_dim >> 1, mode = p.norm_mode;
  const int nq = mode == 1 ? H * D : (mode == 2 ? D : 0), nk = mode == 1 ? Kh * D : nq;
  float* s_qk = s_mem;
  float* s_nw = s_qk + C;                           // [q weights | k weights], of a head or of all
  float* s_sincos = s_nw + nq + nk;
  const int t = blockIdx.x, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, n_warps = nt >> 5;
  const int pos = p.tok_pos[t], slot = p.tok_slot[t];
  const bool conv = p.conv_w != nullptr;
  const int pos0 = conv && p.tok_first != nullptr ? p.tok_pos[p.tok_first[t]] : pos;     // the run's first position
  const int64_t page0 = rb_page_offset(cache, slot, pos, 0), page_step = (int64_t)cache.page_size * Dc;
  for (int i = tid; i < nq + nk; i += nt) s_nw[i] = i < nq ? p.q_norm_w[i] : p.k_norm_w[i - nq];
  for (int i = tid; i < rhalf; i += nt) angle_sincos(pos, p.freq[i], p.magnitude, &s_sincos[i], &s_sincos[rhalf + i]);
  rb_pdl_wait();
  const float* row = p.proj + (int64_t)t * p.ld;
  const int g_at = C + (p.values_are_keys ? 0 : Kh * Dv);
  const int Dc4 = Dc >> 2, own_quads = p.values_are_keys ? 0 : Kh * Dc4;
  auto value_quad = [&](int i, float (&y)[4]) {
    const int kvh = i / Dc4, e = (i - kvh * Dc4) << 2;
    y[0] = y[1] = y[2] = y[3] = 0.f;
    if (e >= Dv) return;
    rb_load4(row + C + kvh * Dv + e, y);
    if (p.mix_rows != nullptr) {
      float other[4];
      rb_load4(p.mix_rows + (int64_t)t * p.mix_ld + kvh * Dv + e, other);
#pragma unroll
      for (int k = 0; k < 4; ++k) y[k] = (1.0f - p.mix_weight) * y[k] + p.mix_weight * other[k];
    }
  };
  T* vdst = (T*)cache.v + page0;
  auto value_to = [&](int i) {
    const int kvh = i / Dc4;
    return vdst + kvh * page_step + ((i - kvh * Dc4) << 2);
  };
  float v0[4], g0 = 0.f;
  if (tid < own_quads) value_quad(tid, v0);
  if (p.gate_heads && tid < H) g0 = row[g_at + tid];
  const float* before[3];
  if (conv) {
#pragma unroll
    for (int back = 1; back <= 3; ++back) {
      const int at = pos - back;
      before[back - 1] = at < 0 ? nullptr : (at >= pos0 ? row - (int64_t)back * p.ld : p.tail + ((int64_t)slot * 4 + (at & 3)) * C);
    }
  }
  float sum_q = 0.f, sum_k = 0.f;
  for (int c = 4 * tid; c < C; c += 4 * nt) {
    float own[4], y[4];
    rb_load4(row + c, own);
    if (conv) {
      float taps[4][4], old[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) rb_load4(p.conv_w + (int64_t)(c + j) * 4, taps[j]);
#pragma unroll
      for (int back = 0; back < 3; ++back)
        if (before[back] != nullptr) rb_load4(before[back] + c, old[back]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[j] = taps[j][3] * own[j];
#pragma unroll
        for (int back = 0; back < 3; ++back)
          if (before[back] != nullptr) y[j] = fmaf(taps[j][2 - back], old[back][j], y[j]);
      }
      if (p.tok_first == nullptr) rb_store4(p.tail + ((int64_t)slot * 4 + (pos & 3)) * C + c, own);      // a row that is its own run
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] = own[j];
    }
    rb_store4(s_qk + c, y);
    const float ss = y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3];
    if (c < H * D) sum_q += ss;
    else sum_k += ss;
  }
  if (tid < own_quads) rb_store4(value_to(tid), v0);
  if (p.gate_heads && tid < H) gates_out[(int64_t)t * H + tid] = rb_from_float<T>(g0);
  if (mode == 1) {
    sum_q = rb_warp_sum(sum_q);
    sum_k = rb_warp_sum(sum_k);
    if (lane == 0) {
      s_sum[0][warp] = sum_q;
      s_sum[1][warp] = sum_k;
    }
  }
  __syncthreads();
  float rq = 1.f, rk = 1.f;
  if (mode == 1) {
    rq = 1.0f / sqrtf(rb_warp_sum(lane < n_warps ? s_sum[0][lane] : 0.f) / (float)(H * D) + p.eps);
    rk = 1.0f / sqrtf(rb_warp_sum(lane < n_warps ? s_sum[1][lane] : 0.f) / (float)(Kh * D) + p.eps);
  }
  const bool apart = !p.interleaved && (rhalf & 3) == 0, within = p.interleaved && (p.rot_dim & 3) == 0;
  for (int head = warp; head < H + Kh; head += n_warps) {
    const bool is_q = head < H;
    T* dst = is_q ? q_out + ((int64_t)t * H + head) * Dc : (T*)cache.k + page0 + (head - H) * page_step;
    const float* src = s_qk + head * D;
    const float* nw = s_nw + (is_q ? 0 : nq) + (mode == 1 ? (is_q ? head : head - H) * D : 0);
    float fac = is_q ? rq : rk;
    if (mode == 2) {
      float ss = 0.f;
      for (int e = 4 * lane; e < D; e += 128) {
        float y[4];
        rb_load4(src + e, y);
        ss += y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3];
      }
      fac = 1.0f / sqrtf(rb_warp_sum(ss) / (float)D + p.eps);
    }
    auto val = [&](int i) { return mode ? src[i] * fac * nw[i] : src[i]; };
    auto quad = [&](int e, float (&y)[4]) {
      rb_load4(src + e, y);
      if (mode) {
        float w[4];
        rb_load4(nw + e, w);
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = y[k] * fac * w[k];
      }
    };
    for (int e = 4 * lane; e < Dc; e += 128) {
      float y[4] = {0.f, 0.f, 0.f, 0.f};
      if (e < p.rot_dim && apart) {                 // the other halves of four pairs are neighbours too
        float me[4], other[4], sn[4], cs[4];
        const bool first = e < rhalf;
        const int pair = first ? e : e - rhalf;
        quad(e, me);
        quad(first ? e + rhalf : pair, other);
        rb_load4(s_sincos + pair, sn);
        rb_load4(s_sincos + rhalf + pair, cs);
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = first ? me[k] * cs[k] - other[k] * sn[k] : me[k] * cs[k] + other[k] * sn[k];
      } else if (e < p.rot_dim && within) {         // two whole pairs
        float me[4];
        quad(e, me);
#pragma unroll
        for (int k = 0; k < 4; k += 2) {
          const float sn = s_sincos[(e + k) >> 1], cs = s_sincos[rhalf + ((e + k) >> 1)];
          y[k] = me[k] * cs - me[k + 1] * sn;
          y[k + 1] = me[k + 1] * cs + me[k] * sn;
        }
      } else if (e < p.rot_dim) {
#pragma unroll
        for (int k = 0; k < 4; ++k) y[k] = turned(val, e + k, p.rot_dim, p.interleaved, s_sincos);
      } else if (e < D) {
        quad(e, y);
      }
      rb_store4(dst + e, y);
    }
  }
  for (int i = tid + nt; i < own_quads; i += nt) {
    value_quad(i, v0);
    rb_store4(value_to(i), v0);
  }
  if (p.values_are_keys)
    for (int i = tid; i < Kh * Dc4; i += nt) {
      const int kvh = i / Dc4, e = (i - kvh * Dc4) << 2;
      float y[4] = {0.f, 0.f, 0.f, 0.f};
      if (e < D) rb_load4(s_qk + (H + kvh) * D + e, y);
      rb_store4(value_to(i), y);
    }
  if (p.gate_heads)
    for (int h = tid + nt; h < H; h += nt) gates_out[(int64_t)t * H + h] = rb_from_float<T>(row[g_at + h]);
}

// A block per token.  rows: [H heads of (D + R) | C latent | R shared key part].  q_out [T, H (D + R)]; the cache row
// (one stream, one head, Dc wide) takes [c / rms(c) * w | turned key part | zeros].
template <typename T>
__global__ void __launch_bounds__(1024) latent_rotate_append_kernel(
    T* q_out, const float* rows, int64_t ld, const float* w, float eps,
    const double* freq, float magnitude, int interleaved, const int* tok_pos,
    const int* tok_slot, RbPagedLayer cache, int H, int D, int R, int C) {
  rb_pdl_launch_dependents();
  __shared__ float scratch[33];
  extern __shared__ float s_sincos[];
  const int t = blockIdx.x;
  const int pos = tok_pos[t], slot = tok_slot[t];
  T* dst = (T*)cache.k + rb_page_offset(cache, slot, pos, 0);
  const float my_w = (int)threadIdx.x < C ? w[threadIdx.x] : 0.f;      // (weights and pages: no kernel of the step writes them)
  for (int i = threadIdx.x; i < R / 2; i += blockDim.x) angle_sincos(pos, freq[i], magnitude, &s_sincos[i], &s_sincos[R / 2 + i]);
  rb_pdl_wait();
  const float* row = rows + (int64_t)t * ld;
  const int Dq = D + R, Dc = cache.head_dim;
  const float* lat = row + (int64_t)H * Dq;
  float ss = 0.f;
  for (int e = threadIdx.x; e < C; e += blockDim.x) ss += lat[e] * lat[e];
  ss = rb_block_sum_once(ss, scratch);                       // also the barrier after the table's writes
  const float r = 1.0f / sqrtf(ss / (float)C + eps);
#pragma unroll 3
  for (int idx = threadIdx.x; idx < H * Dq; idx += blockDim.x) {
    const int head = idx / Dq, e = idx - head * Dq;
    const float* src = row + (int64_t)head * Dq;
    float y;
    if (e < D) {
      y = src[e];
    } else {
      auto val = [&](int i) { return src[D + i]; };
      y = turned(val, e - D, R, interleaved, s_sincos);
    }
    q_out[(int64_t)t * H * Dq + idx] = rb_from_float<T>(y);
  }
  for (int e = threadIdx.x; e < Dc; e += blockDim.x) {
    float y = 0.f;
    if (e < C) {
      y = lat[e] * r * (e == (int)threadIdx.x ? my_w : w[e]);
    } else if (e < C + R) {
      auto val = [&](int i) { return lat[C + i]; };
      y = turned(val, e - C, R, interleaved, s_sincos);
    }
    dst[e] = rb_from_float<T>(y);
  }
}

// rows[t, col0 + head * D + e], head < n_heads: the first rot_dim values of every head turned by the row's position,
// in place.  A block per token; a thread owns whole pairs, so nothing is read after it was written.
__global__ void __launch_bounds__(256) rotate_rows_kernel(float* rows, int64_t ld, int col0, int n_heads, int D,
                                                          const double* freq, float magnitude, int rot_dim,
                                                          int interleaved, const int* tok_pos) {
  rb_pdl_launch_dependents();
  extern __shared__ float s_sincos[];
  const int t = blockIdx.x;
  const int pos = tok_pos[t];
  const int rhalf = rot_dim / 2;
  for (int i = threadIdx.x; i < rhalf; i += blockDim.x) angle_sincos(pos, freq[i], magnitude, &s_sincos[i], &s_sincos[rhalf + i]);
  __syncthreads();
  rb_pdl_wait();
  float* row = rows + (int64_t)t * ld + col0;
  for (int idx = threadIdx.x; idx < n_heads * rhalf; idx += blockDim.x) {
    const int head = idx / rhalf, pair = idx - head * rhalf;
    const int ia = interleaved ? 2 * pair : pair, ib = interleaved ? 2 * pair + 1 : pair + rhalf;
    float* hp = row + (int64_t)head * D;
    const float a = hp[ia], b = hp[ib];
    const float sn = s_sincos[pair], cs = s_sincos[rhalf + pair];
    hp[ia] = a * cs - b * sn;
    hp[ib] = b * cs + a * sn;
  }
}

inline int blocks_for(int64_t n, int threads) {
  const int64_t most = (int64_t)rb_sm_count() * 16;
  const int64_t b = (n + threads - 1) / threads;
  return (int)(b < 1 ? 1 : (b < most ? b : most));
}

}  // namespace

RB_EXPORT int rb_round_rows(void* out, int out_dtype, const float* x, int64_t n, cudaStream_t stream) {
  if (n == 0) return 0;
  if (out_dtype == RB_BF16)
    RB_LAUNCH("round_rows_kernel", (round_rows_kernel<__nv_bfloat16>), blocks_for((n + 3) / 4, 256), 256, 0, stream, (__nv_bfloat16*)out, x, n);
  else if (out_dtype == RB_F32)
    RB_LAUNCH("round_rows_kernel", (round_rows_kernel<float>), blocks_for((n + 3) / 4, 256), 256, 0, stream, (float*)out, x, n);
  else
    RB_FAIL("rb_round_rows: unknown dtype %d", out_dtype);
  RB_CHECK_LAUNCH("rb_round_rows");
  return 0;
}

// x [T, E] += y / rms(y) * w; rounded (or null): the new x in rounded_dtype.
RB_EXPORT int rb_norm_add(float* x, const float* y, const float* w, float eps, int T, int E, void* rounded, int rounded_dtype,
                          cudaStream_t stream) {
  if (T == 0) return 0;
  RB_REQUIRE(E > 0, "rb_norm_add: bad width %d", E);
  const bool wide = E % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)w % 16 == 0;
  const bool vec = wide && E <= 16384 && (uintptr_t)rounded % 16 == 0;        // (more than 16 values a thread do not fit its registers)
  const int n4 = E / 4, nv = n4 <= 256 ? 1 : (n4 <= 1024 ? 2 : 4);
  const int threads = vec ? ((n4 + nv - 1) / nv + 31) / 32 * 32 : (E >= 1024 ? 256 : 128);
#define GO(TT, V, N) RB_LAUNCH("norm_add_kernel", (norm_add_kernel<TT, V, N>), T, threads, 0, stream, x, y, w, eps, E, (TT*)rounded)
#define PICK(TT)                         \
  do {                                   \
    if (!wide) GO(TT, false, 1);         \
    else if (!vec) GO(TT, false, 0);     \
    else if (nv == 1) GO(TT, true, 1);   \
    else if (nv == 2) GO(TT, true, 2);   \
    else GO(TT, true, 4);                \
  } while (0)
  if (rounded == nullptr || rounded_dtype == RB_F32) PICK(float);
  else if (rounded_dtype == RB_BF16) PICK(__nv_bfloat16);
  else RB_FAIL("rb_norm_add: unknown dtype %d", rounded_dtype);
#undef PICK
#undef GO
  RB_CHECK_LAUNCH("rb_norm_add");
  return 0;
}

// x [T, E] += y / rms(y) * w (fresh: x = that; x is then only written), and h [T, E] = x / rms(x) * w2 of the new rows.
RB_EXPORT int rb_norm_add_norm(float* x, const float* y, const float* w, float eps, int T, int E, int fresh, void* h, int h_dtype,
                               const float* w2, float eps2, cudaStream_t stream) {
  if (T == 0) return 0;
  RB_REQUIRE(E > 0 && h != nullptr && w2 != nullptr, "rb_norm_add_norm: bad arguments (width %d)", E);
  RB_REQUIRE(h_dtype == RB_F32 || h_dtype == RB_BF16, "rb_norm_add_norm: unknown dtype %d", h_dtype);
  const bool vec = E % 4 == 0 && E <= 16384 && (uintptr_t)x % 16 == 0 && (uintptr_t)y % 16 == 0 && (uintptr_t)w % 16 == 0 &&
                   (uintptr_t)w2 % 16 == 0 && (uintptr_t)h % 16 == 0;
  const int n4 = E / 4;
  const int nv = n4 <= 256 ? 1 : (n4 <= 1024 ? 2 : 4);
  const int threads = vec ? ((n4 + nv - 1) / nv + 31) / 32 * 32 : 256;
#define GO(TT, V, N, A) RB_LAUNCH("norm_add_norm_kernel", (norm_add_norm_kernel<TT, V, N, A>), T, threads, 0, stream, x, y, w, eps, E, fresh, (TT*)h, w2, eps2)
#define PICK(TT)                                                \
  do {                                                          \
    if (!vec) GO(TT, false, 1, false);                          \
    else if (nv == 1) GO(TT, true, 1, true);                    \
    else if (nv == 2) GO(TT, true, 2, true);                    \
    else if (T <= rb_sm_count()) GO(TT, true, 4, true);         \
    else GO(TT, true, 4, false);                                \
  } while (0)
  if (h_dtype == RB_F32) PICK(float);
  else PICK(__nv_bfloat16);
#undef PICK
#undef GO
  RB_CHECK_LAUNCH("rb_norm_add_norm");
  return 0;
}

// out [T, dim] = gelu_tanh(a[t, :dim]) * table[ids[t], :dim]
RB_EXPORT int rb_token_gate(void* out, int out_dtype, const float* a, int64_t lda, const void* table, int table_dtype,
                            const int* ids, int T, int dim, cudaStream_t stream) {
  if (T == 0) return 0;
  const int64_t n = (int64_t)T * dim;
  const int blocks = blocks_for(n, 256);
#define GO(TO, TT) RB_LAUNCH("token_gate_kernel", (token_gate_kernel<TO, TT>), blocks, 256, 0, stream, (TO*)out, a, lda, (const TT*)table, ids, n, dim)
  if (out_dtype == RB_BF16 && table_dtype == RB_BF16) GO(__nv_bfloat16, __nv_bfloat16);
  else if (out_dtype == RB_F32 && table_dtype == RB_F32) GO(float, float);
  else RB_FAIL("rb_token_gate: unsupported dtypes %d, %d", out_dtype, table_dtype);
#undef GO
  RB_CHECK_LAUNCH("rb_token_gate");
  return 0;
}

// single: every row is a sequence of its own (one launch); else one launch makes the rows and a second moves
// `previous` (int [n_slots]) on to each run's last token.
RB_EXPORT int rb_embed_pairs(float* out, const void* table, const void* pairs, int table_dtype, const int* ids,
                             const int* tok_pos, const int* tok_slot, int* previous, int T, int E, int V, float scale,
                             int buckets, int mul_prev, int mul_cur, int single, cudaStream_t stream) {
  if (T == 0) return 0;
  RB_REQUIRE(E > 0 && V > 0 && buckets > 0 && mul_prev >= 0 && mul_cur >= 0, "rb_embed_pairs: bad sizes E=%d V=%d buckets=%d", E, V, buckets);
  const int threads = E >= 1024 ? 256 : 128;
#define GO(TT, ADD, UPD, THREADS)                                                                                           \
  RB_LAUNCH("embed_pairs_kernel", (embed_pairs_kernel<TT>), T, THREADS, 0, stream, out, (const TT*)table, (const TT*)pairs, ids, \
            tok_pos, tok_slot, previous, T, E, V, scale, buckets, mul_prev, mul_cur, ADD, UPD, single)
  if (table_dtype == RB_BF16) {
    if (single) GO(__nv_bfloat16, 1, 1, threads); else { GO(__nv_bfloat16, 1, 0, threads); GO(__nv_bfloat16, 0, 1, 32); }
  } else if (table_dtype == RB_F32) {
    if (single) GO(float, 1, 1, threads); else { GO(float, 1, 0, threads); GO(float, 0, 1, 32); }
  } else {
    RB_FAIL("rb_embed_pairs: unknown dtype %d", table_dtype);
  }
#undef GO
  RB_CHECK_LAUNCH("rb_embed_pairs");
  return 0;
}

// proj: float32 rows [q (H D) | k (Kh D) | v (Kh Dv), unless values_are_keys | gates (H), if gate_heads].
// dtype: of q_out [T, H, Dc], gates_out [T, H] and the cache.  conv_w: [(H + Kh) D, K] or null; tail: the ring
// [n_slots, K, (H + Kh) D] of a sequence's last projected rows by position modulo K (a step of runs of several rows
// moves it on with rb_conv_tail_update afterwards; tok_first null: every row is its own run and moves it on here).
// norm_mode 1: q and k each under an RMS norm over the whole projection, weights [H D] and [Kh D]; 2: every head
// under its own, one weight [D] for all q heads and one for all k heads; both before the rotation.
RB_EXPORT int rb_qk_prepare(void* q_out, void* gates_out, int dtype, const float* proj, int64_t ld, const float* conv_w, int K,
                            float* tail, const int* tok_first, int norm_mode, const float* q_norm_w, const float* k_norm_w,
                            float eps, const double* freq, float magnitude, int rot_dim, int interleaved, const int* tok_pos,
                            const int* tok_slot, void* cache_k, void* cache_v, const int* page_table, int max_pages,
                            int page_size, int T, int H, int Kh, int D, int Dv, int Dc, int values_are_keys,
                            const float* mix_rows, int64_t mix_ld, float mix_weight, int gate_heads, cudaStream_t stream) {
  if (T == 0) return 0;
  RB_REQUIRE(H > 0 && Kh > 0 && D > 0 && Dv > 0 && Dc >= D && Dc >= Dv && page_size > 0,
             "rb_qk_prepare: bad sizes H=%d Kh=%d D=%d Dv=%d cache width %d", H, Kh, D, Dv, Dc);
  RB_REQUIRE(rot_dim >= 0 && rot_dim <= D && rot_dim % 2 == 0 && (rot_dim == 0 || freq != nullptr),
             "rb_qk_prepare: the rotated prefix %d must be even and at most the head size %d", rot_dim, D);
  RB_REQUIRE(norm_mode == 0 || (q_norm_w != nullptr && k_norm_w != nullptr), "rb_qk_prepare: norm %d without weights", norm_mode);
  RB_REQUIRE(!values_are_keys || Dv == D, "rb_qk_prepare: values that are the keys have the keys' size");
  RB_REQUIRE(conv_w == nullptr || K <= 1 || tail != nullptr, "rb_qk_prepare: a convolution of %d taps needs the ring", K);
  RB_REQUIRE(!gate_heads || gates_out != nullptr, "rb_qk_prepare: gates without a place for them");
  QkParams p{proj, ld, conv_w, K, tail, tok_first, norm_mode, q_norm_w, k_norm_w, eps, freq, magnitude, rot_dim, interleaved,
             tok_pos, tok_slot, H, D, Dv, values_are_keys, mix_rows, mix_ld, mix_weight, gate_heads, 0};
  RbPagedLayer c{cache_k, cache_v, page_table, max_pages, page_size, Kh, Dc};
  const size_t weights = norm_mode == 1 ? (size_t)(H + Kh) * D : (norm_mode == 2 ? (size_t)2 * D : 0);
  size_t smem = ((size_t)rot_dim + (size_t)(H + Kh) * D + (size_t)(H + Kh)) * sizeof(float);
  // (also where it leaves an SM one block: norms of all heads' values, 104 heads of 128, 104 KB with the weights: 1 token 6.5 us, 10.3
  // unstaged, 2,000 146, 178; 176 heads, 176 KB: 8.8, 14.4, 196, 487)
  if (smem + weights * sizeof(float) <= 200 * 1024) { smem += weights * sizeof(float); p.staged = 1; }
  // few tokens (a decode step): a token's block is the whole chain, so it gets as many threads as it has pairs of
  // values to make; many tokens: blocks of 256, several of which share an SM
  int threads = 256;
  if (T <= 2 * rb_sm_count()) {
    const int pairs = (H + Kh) * Dc / 2;
    threads = pairs >= 1024 ? 1024 : (pairs >= 512 ? 512 : 256);
  }
  RB_REQUIRE(smem <= 200 * 1024, "rb_qk_prepare: %d q and k values per token do not fit shared memory", (H + Kh) * D);
  // quads where all sizes, strides and addresses allow it.  Few tokens: a thread for every quad; many: one for five, so that an SM
  // holds more tokens, each of them the whole chain (1,901 tokens of 20 heads of 128: 44 us with a thread a quad, 24.6 with one for
  // two, 19.5 with one for five)
  const uintptr_t all = (uintptr_t)proj | (uintptr_t)q_out | (uintptr_t)cache_k | (uintptr_t)cache_v | (uintptr_t)conv_w |
                        (conv_w != nullptr ? (uintptr_t)tail : 0) | (uintptr_t)mix_rows;
  const bool quads = (D | Dv | Dc) % 4 == 0 && ld % 4 == 0 && (mix_rows == nullptr || mix_ld % 4 == 0) && all % 16 == 0 &&
                     (conv_w == nullptr || K == 4) && (norm_mode == 0 || p.staged);
  if (quads) {
    const int n4 = (H + Kh) * D / 4, want = T <= 2 * rb_sm_count() ? n4 : (n4 + 4) / 5;
    threads = want >= 1024 ? 1024 : (want <= 128 ? 128 : (want + 31) / 32 * 32);
  }
#define GO_AS(NAME, KERNEL)                                                                              \
  do {                                                                                                   \
    if (smem > 48 * 1024)                                                                                \
      RB_CUDA(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));     \
    RB_LAUNCH(NAME, (KERNEL), T, threads, smem, stream, (decltype(q))q_out, (decltype(q))gates_out, p, c); \
  } while (0)
#define GO(TT)                                                                 \
  do {                                                                         \
    TT* q = nullptr;                                                           \
    if (quads) GO_AS("qk_prepare_quads_kernel", qk_prepare_quads_kernel<TT>);  \
    else GO_AS("qk_prepare_kernel", qk_prepare_kernel<TT>);                    \
    (void)q;                                                                   \
  } while (0)
  if (dtype == RB_BF16) GO(__nv_bfloat16);
  else if (dtype == RB_F32) GO(float);
  else RB_FAIL("rb_qk_prepare: unknown dtype %d", dtype);
#undef GO
#undef GO_AS
  RB_CHECK_LAUNCH("rb_qk_prepare");
  return 0;
}

RB_EXPORT int rb_latent_rotate_append(void* q_out, int dtype, const float* rows, int64_t ld, const float* w, float eps,
                                      const double* freq, float magnitude, int interleaved, const int* tok_pos,
                                      const int* tok_slot, void* cache, const int* page_table, int max_pages, int page_size,
                                      int Dc, int T, int H, int D, int R, int C, cudaStream_t stream) {
  if (T == 0) return 0;
  RB_REQUIRE(H > 0 && D > 0 && C > 0 && R >= 0 && R % 2 == 0 && Dc >= C + R && page_size > 0,
             "rb_latent_rotate_append: bad sizes H=%d D=%d R=%d C=%d cache width %d", H, D, R, C, Dc);
  RB_REQUIRE(R == 0 || freq != nullptr, "rb_latent_rotate_append: a turned part without frequencies");
  RbPagedLayer c{cache, cache, page_table, max_pages, page_size, 1, Dc};
  const size_t smem = (size_t)(R > 0 ? R : 1) * sizeof(float);
  // few tokens: a token's block is the whole chain (1 token, 16 heads of 128 + a latent of 128: 4.7 us of a step with 256 threads,
  // 2.8 with 1,024, the page and the weights asked for before the wait)
  const int threads = T <= rb_sm_count() && H * (D + R) >= 2048 ? 1024 : 256;
#define GO(TT) RB_LAUNCH("latent_rotate_append_kernel", (latent_rotate_append_kernel<TT>), T, threads, smem, stream, (TT*)q_out, rows, ld, w, eps, freq, magnitude, interleaved, tok_pos, tok_slot, c, H, D, R, C)
  if (dtype == RB_BF16) GO(__nv_bfloat16);
  else if (dtype == RB_F32) GO(float);
  else RB_FAIL("rb_latent_rotate_append: unknown dtype %d", dtype);
#undef GO
  RB_CHECK_LAUNCH("rb_latent_rotate_append");
  return 0;
}

RB_EXPORT int rb_rotate_rows(float* rows, int64_t ld, int col0, int n_heads, int D, const double* freq, float magnitude,
                             int rot_dim, int interleaved, const int* tok_pos, int T, cudaStream_t stream) {
  if (T == 0 || rot_dim == 0) return 0;
  RB_REQUIRE(n_heads > 0 && D > 0 && rot_dim % 2 == 0 && rot_dim <= D && freq != nullptr,
             "rb_rotate_rows: bad sizes heads=%d D=%d rotated %d", n_heads, D, rot_dim);
  RB_LAUNCH("rotate_rows_kernel", (rotate_rows_kernel), T, 256, (size_t)rot_dim * sizeof(float), stream, rows, ld, col0, n_heads,
            D, freq, magnitude, rot_dim, interleaved, tok_pos);
  RB_CHECK_LAUNCH("rb_rotate_rows");
  return 0;
}

RB_CHECK_READER(prepare)
