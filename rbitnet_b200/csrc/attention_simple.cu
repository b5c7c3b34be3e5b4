// Plain attention over the paged cache for float32 and for any shape the tiled kernels refuse (odd head sizes, pages that
// are no multiple of 64).
//
// Token t at position p of its sequence attends keys max(0, p-window+1)..p of
// its own slot (and, with keep_first, the first keys whatever the window); query head h reads kv head h / (H/Kh); the score is
// (q.k) * scale with the scale applied to the finished dot product; softmax is
// max-subtracted.  crates/bitnet-core/src/llama/model.rs:260-289, :102-114
//
// A group of 8, 16 or 32 lanes (by the head size) takes a key: a lane's share of a row is then a few 16-byte loads and a
// score costs three to five exchanges.  A warp's groups take neighbouring keys, two a turn, each with a running maximum,
// sum and weighted values of its own (all float32), which are joined at the end: the chain from key to key is 4 to 8 times
// shorter than with a warp per key, and a turn's four rows are asked for together.  Where (token, head) pairs are too few
// to give every SM sixteen warps (a decode step), 2, 4 or 8 warps of a block share the keys of a pair.  The order of the
// sums depends on the number of warps that share a pair, so on the number of rows of the step.
// What bounds it is the exchanges and exponentials between the multiply-adds.  One B200, us, a warp per key before and now:
// 32 heads of 64 on 4 kv heads: prompts of 300, 37 and 200 tokens 302, 110; 2,048 tokens 7,409, 2,847; a decode step of 3
// sequences at 300 positions 161, 7.8, of 8 at 2,048 positions 1,094, 30; 32 heads of 128: 8 at 2,048 2,233, 81.
#include "rb_common.cuh"

namespace {

constexpr int WARPS = 8, TURN = 2;

template <typename T, bool VEC, int L>
__device__ __forceinline__ int dim_of(int g, int e, int j) { return VEC ? (g + L * e) * 4 + j : g + L * (4 * e + j); }

template <typename T, bool VEC, int L, int Q>
__device__ __forceinline__ void load_row(const T* row, int g, int D, float (&v)[Q][4]) {
#pragma unroll
  for (int e = 0; e < Q; ++e) {
    if (VEC) {
      if (dim_of<T, VEC, L>(g, e, 0) < D) rb_load4(row + dim_of<T, VEC, L>(g, e, 0), v[e]);
      else v[e][0] = v[e][1] = v[e][2] = v[e][3] = 0.f;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int d = dim_of<T, VEC, L>(g, e, j);
        v[e][j] = d < D ? rb_to_float<T>(row[d]) : 0.f;
      }
    }
  }
}
// what a sum with maximum `m` is multiplied by when the maximum becomes `to`; a sum without keys (maximum -inf) counts nothing
__device__ __forceinline__ float rescale(float m, float to) { return m == -INFINITY ? 0.f : expf(m - to); }

// L lanes a key, Q groups of four values a lane; `share` warps of the block for a (token, head) pair.
template <typename T, bool VEC, int L, int Q>
__global__ void __launch_bounds__(WARPS * 32) attn_simple_kernel(T* out, const T* q,
                                                         RbPagedLayer cache, int page_shift, const int* tok_pos,
                                                         const int* tok_slot, int n_tokens, int H,
                                                         float scale, int window, const float* sinks,
                                                         float softcap, int keep, int share) {
  constexpr int KEYS = 32 / L;
  extern __shared__ float parts[];                     // share > 1: [WARPS][D + 2]
  rb_pdl_launch_dependents();
  rb_pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane % L;
  const int64_t item = (int64_t)blockIdx.x * (WARPS / share) + warp / share;
  const bool live = item < (int64_t)n_tokens * H;
  const int t = live ? (int)(item / H) : 0, h = live ? (int)(item % H) : 0;
  const int D = cache.head_dim;
  const int kvh = h / (H / cache.n_kv_heads);
  const int pos = tok_pos[t], slot = tok_slot[t];
  const T* Kb = (const T*)cache.k;
  const T* Vb = (const T*)cache.v;
  float qr[Q][4], acc[Q][4];
  load_row<T, VEC, L, Q>(q + ((int64_t)t * H + h) * D, g, D, qr);
#pragma unroll
  for (int e = 0; e < Q; ++e)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[e][j] = 0.f;
  float m = -INFINITY, l = 0.f;
  const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;
  const int lo = window > 0 ? max(0, pos - window + 1) : 0;
  // the first `keep` positions that lie before the window, then the window
  const int n_kept = min(keep, lo);
  const int n = live ? pos - lo + n_kept + 1 : 0;
  const int step = KEYS * share;
  for (int i0 = (warp % share) * KEYS; i0 < n; i0 += TURN * step) {
    float s[TURN], kr[TURN][Q][4], vr[TURN][Q][4];
    bool on[TURN];
#pragma unroll
    for (int u = 0; u < TURN; ++u) {
      const int i = i0 + u * step + lane / L;
      on[u] = i < n;
      const int p = !on[u] ? pos : (i < n_kept ? i : lo + (i - n_kept));    // behind the end: the token's own key, not counted
      const int64_t off = rb_page_offset(cache, page_shift, slot, p, kvh);
      load_row<T, VEC, L, Q>(Kb + off, g, D, kr[u]);
      load_row<T, VEC, L, Q>(Vb + off, g, D, vr[u]);
    }
    float mn = m;
#pragma unroll
    for (int u = 0; u < TURN; ++u) {
      float part = 0.f;
#pragma unroll
      for (int e = 0; e < Q; ++e)
#pragma unroll
        for (int j = 0; j < 4; ++j) part = fmaf(qr[e][j], kr[u][e][j], part);
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      s[u] = part * scale;
      if (softcap > 0.f) s[u] = softcap * tanhf(s[u] * inv_cap);
      if (!on[u]) s[u] = -INFINITY;
      mn = fmaxf(mn, s[u]);
    }
    const float corr = rescale(m, mn);
    l *= corr;
#pragma unroll
    for (int e = 0; e < Q; ++e)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[e][j] *= corr;
#pragma unroll
    for (int u = 0; u < TURN; ++u) {
      const float pe = on[u] ? rescale(s[u], mn) : 0.f;
      l += pe;
#pragma unroll
      for (int e = 0; e < Q; ++e)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[e][j] = fmaf(pe, on[u] ? vr[u][e][j] : 0.f, acc[e][j]);
    }
    m = mn;
  }
  // the groups of the warp
#pragma unroll
  for (int o = L; o < 32; o <<= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
    const float mn = fmaxf(m, m2), c1 = rescale(m, mn), c2 = rescale(m2, mn);
    l = l * c1 + l2 * c2;
#pragma unroll
    for (int e = 0; e < Q; ++e)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[e][j] = acc[e][j] * c1 + __shfl_xor_sync(0xffffffffu, acc[e][j], o) * c2;
    m = mn;
  }
  // the warps that share the pair
  if (share > 1) {
    float* mine = parts + warp * (D + 2);
    if (lane < L) {
#pragma unroll
      for (int e = 0; e < Q; ++e)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int d = dim_of<T, VEC, L>(g, e, j);
          if (d < D) mine[d] = acc[e][j];
        }
      if (lane == 0) { mine[D] = m; mine[D + 1] = l; }
    }
    __syncthreads();
    if (warp % share != 0) return;
    for (int w = 1; w < share; ++w) {
      const float* other = parts + (warp + w) * (D + 2);
      const float m2 = other[D], mn = fmaxf(m, m2), c1 = rescale(m, mn), c2 = rescale(m2, mn);
      l = l * c1 + other[D + 1] * c2;
#pragma unroll
      for (int e = 0; e < Q; ++e)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int d = dim_of<T, VEC, L>(g, e, j);
          acc[e][j] = acc[e][j] * c1 + (d < D ? other[d] : 0.f) * c2;
        }
      m = mn;
    }
  }
  if (!live || lane >= L) return;
  float inv;
  if (sinks != nullptr) {                              // the sink: one more term of the denominator, without a value
    const float mn = fmaxf(m, sinks[h]), c = rescale(m, mn);
    inv = c / (l * c + expf(sinks[h] - mn));
  } else {
    inv = 1.0f / l;                                    // every score -inf: 0 / 0, no keys that could be weighed
  }
  T* op = out + ((int64_t)t * H + h) * D;
#pragma unroll
  for (int e = 0; e < Q; ++e) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = acc[e][j] * inv;
    if (VEC) {
      if (dim_of<T, VEC, L>(g, e, 0) < D) rb_store4(op + dim_of<T, VEC, L>(g, e, 0), v);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (dim_of<T, VEC, L>(g, e, j) < D) op[dim_of<T, VEC, L>(g, e, j)] = rb_from_float<T>(v[j]);
    }
  }
}

template <typename T>
int launch(T* out, const T* q, RbPagedLayer c, const int* tok_pos, const int* tok_slot, int n_tokens, int H,
           float scale, int window, cudaStream_t stream) {
  const RbAttentionOptions opt = rb_attention_take();
  const int D = c.head_dim;
  const int64_t items = (int64_t)n_tokens * H;
  int share = 1;
  while (share < WARPS && items * share < 16 * (int64_t)rb_sm_count()) share *= 2;
  const int per_block = WARPS / share;
  const int64_t blocks = (items + per_block - 1) / per_block;
  RB_REQUIRE(blocks <= 0x7fffffff, "rb_attention_simple: %d tokens: too many for one launch", n_tokens);
  const size_t smem = share > 1 ? (size_t)WARPS * (D + 2) * sizeof(float) : 0;      // 33 KB at most
  int shift = -1;
  for (int b = 0; b < 31; ++b)
    if (c.page_size == 1 << b) shift = b;
  const size_t four = 4 * sizeof(T);
  const bool vec = D % 4 == 0 && (uintptr_t)out % four == 0 && (uintptr_t)q % four == 0 && (uintptr_t)c.k % four == 0 && (uintptr_t)c.v % four == 0;
#define GO(L, Q)                                                                                                       \
  do {                                                                                                                 \
    if (vec) RB_LAUNCH("attn_simple_kernel", (attn_simple_kernel<T, true, L, Q>), (int)blocks, WARPS * 32, smem, stream, out, q, c, shift, tok_pos, tok_slot, n_tokens, H, scale, window, opt.sinks, opt.softcap, opt.keep_first, share); \
    else RB_LAUNCH("attn_simple_kernel", (attn_simple_kernel<T, false, L, Q>), (int)blocks, WARPS * 32, smem, stream, out, q, c, shift, tok_pos, tok_slot, n_tokens, H, scale, window, opt.sinks, opt.softcap, opt.keep_first, share);   \
  } while (0)
  // head sizes up to 1,024: at most 16 values of a row a lane up to 256, 32 beyond
  if (D <= 32) GO(8, 1);
  else if (D <= 64) GO(8, 2);
  else if (D <= 96) GO(8, 3);
  else if (D <= 128) GO(8, 4);
  else if (D <= 192) GO(16, 3);
  else if (D <= 256) GO(16, 4);
  else if (D <= 384) GO(32, 3);
  else if (D <= 512) GO(32, 4);
  else if (D <= 768) GO(32, 6);
  else if (D <= 1024) GO(32, 8);
  else RB_FAIL("rb_attention_simple: head_dim %d exceeds 1024", D);
#undef GO
  RB_CHECK_LAUNCH("rb_attention_simple");
  return 0;
}

}  // namespace

static thread_local RbAttentionOptions t_next_attention;

RbAttentionOptions rb_attention_take() {
  const RbAttentionOptions o = t_next_attention;
  t_next_attention = RbAttentionOptions();
  return o;
}

// For the calling thread's next attention launch (any of the library's attention entry points); see rb_common.cuh.
RB_EXPORT int rb_attention_next(const float* sinks, float softcap, int keep_first) {
  t_next_attention.sinks = sinks;
  t_next_attention.keep_first = keep_first > 0 ? keep_first : 0;
  t_next_attention.softcap = softcap > 0.f ? softcap : 0.f;
  return 0;
}

RB_EXPORT int rb_attention_simple(void* out, const void* q, int dtype, const void* cache_k, const void* cache_v,
                                  const int* page_table, int max_pages, int page_size, const int* tok_pos,
                                  const int* tok_slot, int n_tokens, int H, int Kh, int D, float scale,
                                  int window, cudaStream_t stream) {
  if (n_tokens == 0) return 0;
  RB_REQUIRE(H > 0 && Kh > 0 && H % Kh == 0, "rb_attention_simple: heads %d not a multiple of kv heads %d", H, Kh);
  RB_REQUIRE(D > 0 && D <= 1024, "rb_attention_simple: head_dim %d must be in 1..1024", D);
  RbPagedLayer c{(void*)cache_k, (void*)cache_v, page_table, max_pages, page_size, Kh, D};
  if (dtype == RB_F32)
    return launch<float>((float*)out, (const float*)q, c, tok_pos, tok_slot, n_tokens, H, scale, window, stream);
  if (dtype == RB_BF16)
    return launch<__nv_bfloat16>((__nv_bfloat16*)out, (const __nv_bfloat16*)q, c, tok_pos, tok_slot, n_tokens, H,
                                 scale, window, stream);
  RB_FAIL("rb_attention_simple: unknown dtype %d", dtype);
}

RB_CHECK_READER(attention_simple)
