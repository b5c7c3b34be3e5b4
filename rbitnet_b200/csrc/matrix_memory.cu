// Runs of several tokens through a matrix memory with one decay per head and token, in chunks of 64 tokens:
//
//   m_t = max(f_t + m_(t-1), i_t);  C_t = e^(f_t + m_(t-1) - m_t) C_(t-1) + e^(i_t - m_t) k_t v_t^T;  n_t likewise with k alone
//   o_t = C_t^T q_t / (max(|n_t . q_t|, e^(-m_t)) + floor)
//
// (recurrent.cu has the form that goes token by token.)  Within a chunk that starts from C0, n0 and m0, with F_t the sum of
// the chunk's f up to and including t, p_t = F_t - m_t and u_s = i_s - F_s:
//   C_t = e^(p_t + m0) C0 + sum_{s <= t} e^(p_t + u_s) k_s v_s^T
// so a chunk's outputs are two products of 64 rows, and only the memory itself goes from chunk to chunk:
//   memory_gates_kernel       p, u, m of every token (a warp per run and head; F, p and u in float64: what enters an exponential
//                             is a difference of sums that may be large; it is never above 0 but for m's rounding)
//   memory_chunk_sum_kernel   every chunk's own sum over its tokens, for the memory and for n, and its scores
//                             (q_t . k_s) e^(p_t + u_s), all chunks at once
//   memory_chunk_walk_kernel  the walk over a run's chunks, value by value: leaves in each sum's place what the chunk starts from
//   memory_chunk_out_kernel   every chunk's outputs, all at once
// Every operand, product and sum is float32 (FFMA).  The first form bounds a prompt by its chain of tokens (2,048 tokens of 8
// heads of 128 x 256: 770 us); here the products are bound by the multiply-adds and the shared memory that feeds them, the
// walk by the memory's bytes: gates 57, sums and scores 54, walk 21, outputs 91 us, each launch by itself with cold caches; about
// 210 with the norm in a step (memories of 256 x 512: 1,968 us token by token, 508 in chunks before the sums in groups).
#include "rb_common.cuh"

namespace {

constexpr int CH = 64;                   // tokens of a chunk
constexpr int NT = 128;                  // threads of a product's block: 64 x 64 outputs, 8 x 4 a thread
constexpr int PITCH = CH + 4;

struct Memory {
  const float* proj;                     // float32 rows [q (H D) | k (H D) | v (H Dv) | ...], gates' pre-activations at i_off + h, f_off + h
  int64_t ld;
  int q_off, k_off, v_off, i_off, f_off;
  int H, D, Dv;
  const int *chunk_row, *chunk_len;      // a chunk's first row and its tokens
  float* sums;                           // [chunk][H][Dv D + D]: a chunk's sum, then what it starts from ([value column][row], then n)
  float* scores;                         // [chunk][H][64][64]
  double *p, *u;                         // [chunk][H][64]
  float* m;                              // [chunk][H][64]
  float* m0;                             // [chunk][H]
  int vec;                               // rows, offsets and sizes are multiples of four values, pointers of 16 bytes
  __device__ __forceinline__ int64_t at(int chunk, int h) const { return (int64_t)chunk * H + h; }
  __device__ __forceinline__ int64_t size() const { return (int64_t)Dv * D + D; }
};

// One warp per (run, head), two tokens a lane; the next chunk's pre-activations are on their way while a chunk is worked on.
__global__ void __launch_bounds__(128) memory_gates_kernel(Memory a, const float* i_bias, const float* f_bias,
                                                           float cap, float* m_state, const int* run_chunk0,
                                                           const int* seq_first, const int* seq_count,
                                                           const int* tok_slot) {
  rb_pdl_launch_dependents();
  const int lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (h >= a.H) return;
  const float ib = i_bias != nullptr ? i_bias[h] : 0.f, fb = f_bias != nullptr ? f_bias[h] : 0.f;
  rb_pdl_wait();
  const int n = seq_count[blockIdx.x], first = seq_first[blockIdx.x], slot = tok_slot[first], chunk0 = run_chunk0[blockIdx.x];
  float gi[2], gf[2];
  auto fetch = [&](int t0) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t = t0 + 2 * lane + k;
      gi[k] = gf[k] = 0.f;
      if (t < n) {
        const float* row = a.proj + (int64_t)(first + t) * a.ld;
        gi[k] = row[a.i_off + h];
        gf[k] = row[a.f_off + h];
      }
    }
  };
  fetch(0);
  float m = m_state[(int64_t)slot * a.H + h];
  for (int t0 = 0; t0 < n; t0 += CH) {
    double f[2], i[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bool on = t0 + 2 * lane + k < n;
      const float fc = cap * tanhf((gf[k] + fb) / cap);
      f[k] = on ? (double)(fminf(fc, 0.f) - log1pf(expf(-fabsf(fc)))) : 0.0;             // log sigmoid
      i[k] = on ? (double)(cap * tanhf((gi[k] + ib) / cap)) : -INFINITY;
    }
    if (t0 + CH < n) fetch(t0 + CH);
    const double f1 = f[0] + f[1];
    double F = f1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, F, o);
      if (lane >= o) F += v;
    }
    const double F0 = F - f[1];                                                          // of this lane's two tokens: F0, F
    const double u0 = i[0] - F0, u1 = i[1] - F;
    double G = fmax(u0, u1);                                                             // the greatest u up to the second
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(0xffffffffu, G, o);
      if (lane >= o) G = fmax(G, v);
    }
    double before = __shfl_up_sync(0xffffffffu, G, 1);
    if (lane == 0) before = -INFINITY;
    const float m_a = (float)(F0 + fmax((double)m, fmax(before, u0))), m_b = (float)(F + fmax((double)m, G));
    const int64_t at = a.at(chunk0 + t0 / CH, h);
    const int64_t to = at * CH + 2 * lane;
    a.p[to] = F0 - (double)m_a;
    a.p[to + 1] = F - (double)m_b;
    a.u[to] = u0;
    a.u[to + 1] = u1;
    a.m[to] = m_a;
    a.m[to + 1] = m_b;
    if (lane == 0) a.m0[at] = m;
    m = __shfl_sync(0xffffffffu, m_b, 31);                // (behind the run's end f = 0 and i = -inf leave m as it is)
  }
  if (lane == 0) m_state[(int64_t)slot * a.H + h] = m;
}

// 64 values of `width` (from column c0, `live` in all) of 64 rows, of which `rows` are there, into dst [depth][PITCH].
// TURN: the rows become the columns (depth = the row's values), else a row stays a row.  What is not there is zero; row r
// is multiplied by mul[r] (null: 1).
template <bool TURN>
__device__ __forceinline__ void stage(float* dst, const float* src, int64_t ld, int rows, int c0, int live, bool vec,
                                      const float* mul) {
#pragma unroll 4
  for (int e = threadIdx.x; e < CH * CH / 4; e += NT) {
    const int r = e / (CH / 4), c = e % (CH / 4) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (r < rows) {
      const float* s = src + (int64_t)r * ld + c0 + c;
      if (vec) {
        if (c0 + c < live) rb_load4(s, v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (c0 + c + j < live) v[j] = s[j];
      }
      const float w = mul != nullptr ? mul[r] : 1.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] *= w;
    }
    if (TURN) {
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[(c + j) * PITCH + r] = v[j];
    } else {
      rb_store4(dst + r * PITCH + c, v);
    }
  }
}

// acc[i][j] += sum over k of x[k][row i] y[k][column j]; a thread's rows are 4 ty + {0..3} and 32 + 4 ty + {0..3}, its columns
// 4 tx + {0..3}.  Every 32 products are summed from zero and added once: one chain over k would round each of a value's
// 64 + D products at the size of the whole (D 256: outputs off by 4.3e-7 in one chain, 2.0e-7 so, 2.5e-7 token by
// token; 2,048 tokens of 8 heads of 128 x 256 take 1 % longer).
__device__ __forceinline__ void multiply(float (&acc)[8][4], const float* x, const float* y, int tx, int ty) {
#pragma unroll 1
  for (int k0 = 0; k0 < CH; k0 += 32) {
    float part[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
#pragma unroll 8
    for (int k = k0; k < k0 + 32; ++k) {
      float a[2][4], b[4];
      rb_load4(x + k * PITCH + ty * 4, a[0]);
      rb_load4(x + k * PITCH + 32 + ty * 4, a[1]);
      rb_load4(y + k * PITCH + tx * 4, b);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[i][j] = fmaf(a[i / 4][i % 4], b[j], part[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
  }
}
// The same for x that is zero for k behind the row (a chunk's scores): later tokens are left out of a row's sum and not
// multiplied by zeros, since one of them that is infinite would turn the tokens before it into NaN.
__device__ __forceinline__ void multiply_below(float (&acc)[8][4], const float* x, const float* y, int tx, int ty) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    const int r0 = 32 * g + 4 * ty;                      // this group's first row: every k before it, then k = row by row
    float part[4][4];
    auto clear = [&]() {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
    };
    auto add = [&]() {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[4 * g + i][j] += part[i][j];
    };
    auto take = [&](int k, int first) {
      float a[4], b[4];
      rb_load4(x + k * PITCH + r0, a);
      rb_load4(y + k * PITCH + tx * 4, b);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i >= first) part[i][j] = fmaf(a[i], b[j], part[i][j]);
    };
    clear();
    if (g == 1) {
#pragma unroll 4
      for (int k = 0; k < 32; ++k) take(k, 0);
      add();
      clear();
    }
#pragma unroll 4
    for (int k = 32 * g; k < r0; ++k) take(k, 0);
#pragma unroll
    for (int e = 0; e < 4; ++e) take(r0 + e, e);
    add();
  }
}
__device__ __forceinline__ int row_of(int i, int ty) { return i / 4 * 32 + ty * 4 + i % 4; }

// grid (chunks, H, 1 + tiles of 64 value columns x tiles of 64 rows).  The first z makes the chunk's scores.
__global__ void __launch_bounds__(NT, 5) memory_chunk_sum_kernel(Memory a) {
  rb_pdl_launch_dependents();
  __shared__ __align__(16) float x[CH * PITCH], y[CH * PITCH];
  __shared__ float w[CH];
  const int chunk = blockIdx.x, h = blockIdx.y, tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  rb_pdl_wait();
  const int rows = a.chunk_len[chunk];
  const float* base = a.proj + (int64_t)a.chunk_row[chunk] * a.ld;
  const int64_t at = a.at(chunk, h);
  const double *p = a.p + at * CH, *u = a.u + at * CH;
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  if (blockIdx.z == 0) {
    for (int d0 = 0; d0 < a.D; d0 += CH) {
      stage<true>(x, base + a.q_off + h * a.D, a.ld, rows, d0, a.D, a.vec, nullptr);
      stage<true>(y, base + a.k_off + h * a.D, a.ld, rows, d0, a.D, a.vec, nullptr);
      __syncthreads();
      multiply(acc, x, y, tx, ty);
      __syncthreads();
    }
    float* out = a.scores + at * CH * CH;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = row_of(i, ty);
      const double pt = p[t];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int s = tx * 4 + j;
        acc[i][j] = s <= t && t < rows ? acc[i][j] * expf((float)(pt + u[s])) : 0.f;
      }
      rb_store4(out + t * CH + tx * 4, acc[i]);
    }
    return;
  }
  const int tiles_d = (a.D + CH - 1) / CH;
  const int j0 = (blockIdx.z - 1) / tiles_d * CH, d0 = (blockIdx.z - 1) % tiles_d * CH;
  // a token's weight at the chunk's end; behind the last token u = -inf leaves zero
  if (threadIdx.x < CH) w[threadIdx.x] = expf((float)(p[CH - 1] + u[threadIdx.x]));
  stage<false>(y, base + a.k_off + h * a.D, a.ld, rows, d0, a.D, a.vec, nullptr);
  __syncthreads();
  stage<false>(x, base + a.v_off + h * a.Dv, a.ld, rows, j0, a.Dv, a.vec, w);
  __syncthreads();
  multiply(acc, x, y, tx, ty);
  float* out = a.sums + at * a.size();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int j = j0 + row_of(i, ty), d = d0 + tx * 4;
    if (j >= a.Dv) continue;
    float* to = out + (int64_t)j * a.D + d;
    if (a.vec) {
      if (d < a.D) rb_store4(to, acc[i]);
    } else {
#pragma unroll
      for (int x4 = 0; x4 < 4; ++x4)
        if (d + x4 < a.D) to[x4] = acc[i][x4];
    }
  }
  if (j0 == 0 && threadIdx.x < CH && d0 + threadIdx.x < a.D) {
    float n = 0.f;
    for (int s = 0; s < rows; ++s) n = fmaf(w[s], y[s * PITCH + threadIdx.x], n);
    out[(int64_t)a.Dv * a.D + d0 + threadIdx.x] = n;
  }
}

// grid (runs, H, pieces); V neighbouring values a thread.
template <int V>
__global__ void __launch_bounds__(128) memory_chunk_walk_kernel(Memory a, float* C_state, float* n_state,
                                                                const int* run_chunk0, const int* seq_first,
                                                                const int* seq_count, const int* tok_slot) {
  rb_pdl_launch_dependents();
  rb_pdl_wait();
  const int h = blockIdx.y, chunk0 = run_chunk0[blockIdx.x], chunks = (seq_count[blockIdx.x] + CH - 1) / CH;
  const int64_t slot = tok_slot[seq_first[blockIdx.x]];
  const int64_t i = ((int64_t)blockIdx.z * blockDim.x + threadIdx.x) * V, memory = (int64_t)a.Dv * a.D;
  if (i >= a.size()) return;
  float* state = i < memory ? C_state + (slot * a.H + h) * memory + i : n_state + (slot * a.H + h) * a.D + (i - memory);
  float cur[V];
#pragma unroll
  for (int k = 0; k < V; ++k) cur[k] = state[k];
  constexpr int AHEAD = 4;
  for (int c = 0; c < chunks; c += AHEAD) {
    float in[AHEAD][V], keep[AHEAD];
#pragma unroll
    for (int x = 0; x < AHEAD; ++x) {
      if (c + x < chunks) {
        const int64_t at = a.at(chunk0 + c + x, h);
        keep[x] = expf((float)(a.p[at * CH + CH - 1] + (double)a.m0[at]));
        const float* s = a.sums + at * a.size() + i;
        if constexpr (V == 4) rb_load4(s, in[x]);
        else in[x][0] = s[0];
      }
    }
#pragma unroll
    for (int x = 0; x < AHEAD; ++x) {
      if (c + x < chunks) {
        float* s = a.sums + a.at(chunk0 + c + x, h) * a.size() + i;
        if constexpr (V == 4) rb_store4(s, cur);
        else s[0] = cur[0];
#pragma unroll
        for (int k = 0; k < V; ++k) cur[k] = fmaf(keep[x], cur[k], in[x][k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < V; ++k) state[k] = cur[k];
}

// grid (chunks, H, tiles of 64 value columns): scores x v, then (e^(p_t + m0) q) x what the chunk starts from.
__global__ void __launch_bounds__(NT, 5) memory_chunk_out_kernel(Memory a, float* o_out, float q_scale, float floor_add) {
  rb_pdl_launch_dependents();
  __shared__ __align__(16) float x[CH * PITCH], y[CH * PITCH];
  __shared__ float carry[CH], n0[CH], nq[2][CH];
  const int chunk = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * CH, tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int t = threadIdx.x % CH, half = threadIdx.x / CH;            // a thread's share of n . q: every second k of row t
  rb_pdl_wait();
  const int rows = a.chunk_len[chunk], row0 = a.chunk_row[chunk];
  const float* base = a.proj + (int64_t)row0 * a.ld;
  const int64_t at = a.at(chunk, h);
  const float* start = a.sums + at * a.size();
  if (threadIdx.x < CH) carry[threadIdx.x] = expf((float)(a.p[at * CH + threadIdx.x] + (double)a.m0[at]));
  float acc[8][4], sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  stage<true>(x, a.scores + at * CH * CH, CH, CH, 0, CH, true, nullptr);
  stage<false>(y, base + a.v_off + h * a.Dv, a.ld, rows, j0, a.Dv, a.vec, nullptr);
  __syncthreads();
  multiply_below(acc, x, y, tx, ty);
#pragma unroll 8
  for (int k = half; k < CH; k += 2) sum += x[k * PITCH + t];
  for (int d0 = 0; d0 < a.D; d0 += CH) {
    __syncthreads();
    stage<true>(x, base + a.q_off + h * a.D, a.ld, rows, d0, a.D, a.vec, carry);
    stage<true>(y, start + (int64_t)j0 * a.D, a.D, min(CH, a.Dv - j0), d0, a.D, a.vec, nullptr);
    if (threadIdx.x < CH) n0[threadIdx.x] = d0 + threadIdx.x < a.D ? start[(int64_t)a.Dv * a.D + d0 + threadIdx.x] : 0.f;
    __syncthreads();
    multiply(acc, x, y, tx, ty);
#pragma unroll 8
    for (int k = half; k < CH; k += 2) sum = fmaf(x[k * PITCH + t], n0[k], sum);
  }
  nq[half][t] = sum;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = row_of(i, ty);
    if (r >= rows) continue;
    const float n = nq[0][r] + nq[1][r];
    const float scale = q_scale / (fmaxf(fabsf(n * q_scale), expf(-a.m[at * CH + r])) + floor_add);
    float* to = o_out + ((int64_t)(row0 + r) * a.H + h) * a.Dv + j0 + tx * 4;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] *= scale;
    if (a.vec) {
      if (j0 + tx * 4 < a.Dv) rb_store4(to, acc[i]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j0 + tx * 4 + j < a.Dv) to[j] = acc[i][j];
    }
  }
}

// Blocks of the walk for one (run, head): 128 threads of four values, of one where rows do not allow that.
int64_t walk_pieces(int D, int Dv) {
  const int64_t values = (int64_t)Dv * D + D;
  return ((D % 4 == 0 ? values / 4 : values) + 127) / 128;
}

}  // namespace

// Whether the chunked form takes heads of this size: the blocks of the sums and of the walk for a head are counted in the grid's third
// dimension (33 million values a head; 8 million where D is no multiple of four).
RB_EXPORT int rb_matrix_memory_chunked_takes(int D, int Dv) {
  const int64_t tiles = (((int64_t)Dv + CH - 1) / CH) * ((D + CH - 1) / CH);
  return D > 0 && D <= 512 && Dv > 0 && tiles < 65535 && walk_pieces(D, Dv) <= 65535;
}

// Scratch of the chunked form in floats.
RB_EXPORT long long rb_matrix_memory_chunk_floats(int n_chunks, int H, int D, int Dv) {
  const int64_t heads = (int64_t)n_chunks * H;
  return heads * ((int64_t)Dv * D + D + CH * CH + CH * 5 + 1) + 16;
}

// Runs of several tokens (seq_first, seq_count), cut into chunks of 64: chunk_row, chunk_len, and run_chunk0, a run's first
// chunk.  scratch: rb_matrix_memory_chunk_floats floats, 16-byte aligned.  The rest as in
// rb_matrix_memory.
RB_EXPORT int rb_matrix_memory_chunked(float* o_out, const float* proj, int64_t ld, int q_off, int k_off, int v_off, int i_off,
                                       int f_off, const float* i_bias, const float* f_bias, float cap, float q_scale,
                                       float floor_add, float* C_state, float* n_state, float* m_state, const int* seq_first,
                                       const int* seq_count, const int* run_chunk0, const int* chunk_row, const int* chunk_len,
                                       const int* tok_slot, int n_seq, int n_chunks, int H, int D, int Dv, float* scratch,
                                       cudaStream_t stream) {
  if (n_seq == 0) return 0;
  RB_REQUIRE(H > 0 && H <= 65535 && n_chunks > 0 && rb_matrix_memory_chunked_takes(D, Dv), "rb_matrix_memory_chunked: sizes H=%d D=%d Dv=%d are not taken", H, D, Dv);
  RB_REQUIRE(cap > 0.f, "rb_matrix_memory_chunked: the gates' cap must be positive");
  RB_REQUIRE((uintptr_t)scratch % 16 == 0, "rb_matrix_memory_chunked: scratch must be 16-byte aligned");
  const int64_t heads = (int64_t)n_chunks * H;
  Memory a;
  a.proj = proj; a.ld = ld;
  a.q_off = q_off; a.k_off = k_off; a.v_off = v_off; a.i_off = i_off; a.f_off = f_off;
  a.H = H; a.D = D; a.Dv = Dv;
  a.chunk_row = chunk_row; a.chunk_len = chunk_len;
  a.p = reinterpret_cast<double*>(scratch);
  a.u = a.p + heads * CH;
  a.m = reinterpret_cast<float*>(a.u + heads * CH);
  a.scores = a.m + heads * CH;
  a.sums = a.scores + heads * CH * CH;
  a.m0 = a.sums + heads * ((int64_t)Dv * D + D);
  a.vec = D % 4 == 0 && Dv % 4 == 0 && ld % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 &&
          (uintptr_t)proj % 16 == 0 && (uintptr_t)o_out % 16 == 0 && (uintptr_t)C_state % 16 == 0;
  const int tiles_j = (Dv + CH - 1) / CH, tiles_d = (D + CH - 1) / CH;
  RB_LAUNCH("memory_gates_kernel", (memory_gates_kernel), dim3(n_seq, (H + 3) / 4), 128, 0, stream, a, i_bias, f_bias, cap, m_state,
            run_chunk0, seq_first, seq_count, tok_slot);
  RB_LAUNCH("memory_chunk_sum_kernel", (memory_chunk_sum_kernel), dim3(n_chunks, H, 1 + tiles_j * tiles_d), NT, 0, stream, a);
  const dim3 walk(n_seq, H, (unsigned)walk_pieces(D, Dv));
  if (D % 4 == 0)
    RB_LAUNCH("memory_chunk_walk_kernel", (memory_chunk_walk_kernel<4>), walk, 128, 0, stream, a, C_state, n_state,
              run_chunk0, seq_first, seq_count, tok_slot);
  else
    RB_LAUNCH("memory_chunk_walk_kernel", (memory_chunk_walk_kernel<1>), walk, 128, 0, stream, a, C_state, n_state,
              run_chunk0, seq_first, seq_count, tok_slot);
  RB_LAUNCH("memory_chunk_out_kernel", (memory_chunk_out_kernel), dim3(n_chunks, H, tiles_j), NT, 0, stream, a, o_out, q_scale, floor_add);
  RB_CHECK_LAUNCH("rb_matrix_memory_chunked");
  return 0;
}
