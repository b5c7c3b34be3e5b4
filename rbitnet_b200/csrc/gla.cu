// Gated linear attention: a matrix memory S [key channels, value columns] per head with a decay per key channel,
//
//   S_t = diag(alpha_t) S_(t-1) + k_t v_t^T,     o_t = S_t^T q_t,
//   alpha_t = sigmoid(z_t)^(1/tau),              z_t = A2 (A1 h_t) + b        (a low-rank product, laid out heads x channels)
//
// The memory is float32 and is kept by value column ([slot][head][column][channel]), so that what one thread owns
// is contiguous.  rows: float32 [T, ...] of the mixer's stacked projection, holding q, k, v and A1 h at the given
// columns.  A step's rows of one sequence are a run; the memory is read at a run's start and written at its end.
//
// gla_decay_kernel   alpha for every row and channel: exp(-softplus(-z) / tau), all float32
// gla_scan_kernel    a block per (run, head, tile of value columns).  A column lies on P lanes, each holding R = 16
//                    channels of it in registers; a chunk of rows' q, k and alpha is staged in shared memory for all
//                    the block's columns; per row a lane does R decays, R updates and R products, and log2 P
//                    exchanges finish a column's output.  Token by token: the plain form, and a decode step's: then it
//                    is bound by reading and writing the memory, whose channels the lanes of a column take in neighbouring
//                    groups of four, 16 bytes an access (8 sequences of 8 heads of 128 x 256: 17.5 us a
//                    step with channels p R + r and an access each, 4.9 so).
// gla_chunk_*        runs of several tokens in chunks of 32, the chain in time only from chunk to chunk (below).
// gla_step_kernel    a decode step in one launch: decays, the memory's step, the norm per head and the gate.
#include "rb_common.cuh"

namespace {

constexpr int GLA_R = 16;        // channels a lane holds

__device__ __forceinline__ float softplus_(float v) { return v > 20.f ? v : log1pf(expf(v)); }

// A block takes GLA_DT rows and 128 channels at a time: a channel's row of A2 is read once for all of them.
constexpr int GLA_DT = 8;
__global__ void __launch_bounds__(128) gla_decay_kernel(float* alpha, const float* rows, int64_t ld,
                                                        int a_off, const float* A2,
                                                        const float* bias, int T, int C, int rank,
                                                        float inv_tau, int as_log) {
  rb_pdl_launch_dependents();
  rb_pdl_wait();
  const int t0 = blockIdx.x * GLA_DT, nt = min(GLA_DT, T - t0);
  extern __shared__ float s_low[];                 // A1 h of these rows: [GLA_DT][rank], zeros for rows beyond the last
  for (int e = threadIdx.x; e < GLA_DT * rank; e += blockDim.x) {
    const int i = e / rank, r = e - i * rank;
    s_low[e] = i < nt ? rows[(int64_t)(t0 + i) * ld + a_off + r] : 0.f;
  }
  __syncthreads();
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
    float z[GLA_DT];
    const float b = bias != nullptr ? bias[c] : 0.f;
#pragma unroll
    for (int i = 0; i < GLA_DT; ++i) z[i] = b;
    const float* w = A2 + (int64_t)c * rank;
    for (int r = 0; r < rank; ++r) {
      const float wr = w[r];
#pragma unroll
      for (int i = 0; i < GLA_DT; ++i) z[i] = fmaf(wr, s_low[i * rank + r], z[i]);
    }
#pragma unroll
    for (int i = 0; i < GLA_DT; ++i) {
      if (i < nt) {
        const float lg = -softplus_(-z[i]) * inv_tau;            // log alpha
        alpha[(int64_t)(t0 + i) * C + c] = as_log ? lg : expf(lg);
      }
    }
  }
}

template <int P>
__global__ void __launch_bounds__(128) gla_scan_kernel(float* o, const float* rows, int64_t ld,
                                                       int q_off, int k_off, int v_off, const float* alpha,
                                                       float q_scale, float* state,
                                                       const int* seq_first, const int* seq_count,
                                                       const int* tok_slot, int H, int D, int Dv,
                                                       int64_t a_ld) {
  rb_pdl_launch_dependents();
  constexpr int COLS = 128 / P;                    // value columns of a block
  constexpr int DP = P * GLA_R;                    // channels with padding
  constexpr int GLA_CHUNK = P <= 8 ? 16 : (P == 16 ? 8 : 4);   // rows staged at once: 24 KB of q, k and alpha at most
  __shared__ __align__(16) float s_q[GLA_CHUNK][DP], s_k[GLA_CHUNK][DP], s_a[GLA_CHUNK][DP];
  __shared__ float s_v[GLA_CHUNK][COLS];
  const int run = blockIdx.x, head = blockIdx.y;
  const int col = threadIdx.x / P, p = threadIdx.x % P;
  const int j = blockIdx.z * COLS + col;           // this thread's value column
  rb_pdl_wait();
  const int first = seq_first != nullptr ? seq_first[run] : run;
  const int n = seq_count != nullptr ? seq_count[run] : 1;
  const int slot = tok_slot[first];
  float S[GLA_R];                                  // channels 4 (p + P g) + {0..3}, g = 0..3
  float* mine = state + (((int64_t)slot * H + head) * Dv + j) * D;
  const bool vec = (D & 3) == 0 && ((uintptr_t)state & 15) == 0;
#pragma unroll
  for (int g = 0; g < GLA_R / 4; ++g) {
    const int d = 4 * (p + P * g);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (j < Dv) {
      if (vec) {
        if (d < D) rb_load4(mine + d, v);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (d + i < D) v[i] = mine[d + i];
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) S[4 * g + i] = v[i];
  }
  for (int t0 = 0; t0 < n; t0 += GLA_CHUNK) {
    const int nt = min(GLA_CHUNK, n - t0);
    __syncthreads();
    for (int e = threadIdx.x; e < nt * DP; e += blockDim.x) {
      const int i = e / DP, d = e % DP;
      const int64_t row = (int64_t)(first + t0 + i) * ld;
      const bool in = d < D;
      s_q[i][d] = in ? rows[row + q_off + head * D + d] * q_scale : 0.f;
      s_k[i][d] = in ? rows[row + k_off + head * D + d] : 0.f;
      s_a[i][d] = in ? alpha[(int64_t)(first + t0 + i) * a_ld + head * D + d] : 0.f;
    }
    for (int e = threadIdx.x; e < nt * COLS; e += blockDim.x) {
      const int i = e / COLS, c = e % COLS;
      const int jj = blockIdx.z * COLS + c;
      s_v[i][c] = jj < Dv ? rows[(int64_t)(first + t0 + i) * ld + v_off + head * Dv + jj] : 0.f;
    }
    __syncthreads();
    for (int i = 0; i < nt; ++i) {
      const float v = s_v[i][col];
      float acc = 0.f;
#pragma unroll
      for (int r4 = 0; r4 < GLA_R; r4 += 4) {
        const int d = 4 * p + P * r4;
        const float4 a = *reinterpret_cast<const float4*>(&s_a[i][d]);
        const float4 k = *reinterpret_cast<const float4*>(&s_k[i][d]);
        const float4 q = *reinterpret_cast<const float4*>(&s_q[i][d]);
        S[r4 + 0] = fmaf(a.x, S[r4 + 0], k.x * v); acc = fmaf(S[r4 + 0], q.x, acc);
        S[r4 + 1] = fmaf(a.y, S[r4 + 1], k.y * v); acc = fmaf(S[r4 + 1], q.y, acc);
        S[r4 + 2] = fmaf(a.z, S[r4 + 2], k.z * v); acc = fmaf(S[r4 + 2], q.z, acc);
        S[r4 + 3] = fmaf(a.w, S[r4 + 3], k.w * v); acc = fmaf(S[r4 + 3], q.w, acc);
      }
#pragma unroll
      for (int off = P / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
      if (p == 0 && j < Dv) o[((int64_t)(first + t0 + i) * H + head) * Dv + j] = acc;
    }
  }
  if (j >= Dv) return;
#pragma unroll
  for (int g = 0; g < GLA_R / 4; ++g) {
    const int d = 4 * (p + P * g);
    const float v[4] = {S[4 * g], S[4 * g + 1], S[4 * g + 2], S[4 * g + 3]};
    if (vec) {
      if (d < D) rb_store4(mine + d, v);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (d + i < D) mine[d + i] = v[i];
    }
  }
}

template <int P>
int launch_scan(float* o, const float* rows, int64_t ld, int q_off, int k_off, int v_off, const float* alpha, float q_scale,
                float* state, const int* seq_first, const int* seq_count, const int* tok_slot, int n_runs, int H, int D,
                int Dv, int64_t a_ld, cudaStream_t stream) {
  constexpr int COLS = 128 / P;
  const dim3 grid(n_runs, H, (Dv + COLS - 1) / COLS);
  RB_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "rb_gla_scan: %d heads of %d value columns are too many for one launch", H, Dv);
  RB_LAUNCH("gla_scan_kernel", (gla_scan_kernel<P>), grid, 128, 0, stream, o, rows, ld, q_off, k_off, v_off, alpha, q_scale,
            state, seq_first, seq_count, tok_slot, H, D, Dv, a_ld);
  RB_CHECK_LAUNCH("rb_gla_scan");
  return 0;
}

// ---------------------------------------------------------------- long runs: chunks of 32 tokens
// Within a chunk that starts from the memory S0, with B_i[d] the sum of the logarithms of channel d's decays over the
// chunk's tokens up to and including i (so that exp(B_i - B_j) is the decay from token j to token i, never above one):
//   o_i   = (q_i * e^{B_i})^T S0 + sum_{j <= i} M_ij v_j,      M_ij = sum_d q_i[d] k_j[d] e^{B_i[d] - B_j[d]}
//   S_end = diag(e^{B_end}) S0 + sum_j (k_j * e^{B_end - B_j}) v_j^T
// Every exponent is taken of a difference that is zero or negative, channel by channel, so nothing overflows however
// fast a channel forgets.  The first kernel makes Qt = q e^{B}, Kt = k e^{B_end - B}, M and e^{B_end} for every
// (chunk, head) at once; the second walks a run's chunks with the memory: two small products per chunk.  A chunk's
// missing tokens (the run's end) count as decay 1 and k = q = v = 0.
constexpr int GCH = 32;          // tokens of a chunk
// second kernel, value columns of a block CT: threads (CT / 4 warps on the memory, eight on the outputs) and row stride of the
// memory's tile (a phase of eight lanes reads one row of 32 columns, or two rows four apart of 16: those then begin 16 banks apart)
__host__ __device__ constexpr int gscan_threads(int CT) { return 8 * CT + 256; }
__host__ __device__ constexpr int gscan_stride(int CT) { return CT == 32 ? 32 : CT + 4; }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16_or_zeros(void* dst, const void* src, bool real) {
  const int bytes = real ? 16 : 0;            // fewer source bytes than 16: the rest is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__host__ __device__ constexpr int gla_item_floats(int D) { return 2 * GCH * D + GCH * GCH + D; }   // Qt, Kt, M, e^{B_end}

// grid (chunks, H), 128 threads.  log_alpha: [T, H * D].  Scratch per (chunk, head): Qt [32][D], Kt [32][D], M [32][32],
// e^{B_end} [D].
__global__ void __launch_bounds__(128) gla_chunk_prepare_kernel(float* scratch, const float* rows,
                                                                int64_t ld, int q_off, int k_off,
                                                                const float* log_alpha, float q_scale,
                                                                const int* chunk_row,
                                                                const int* chunk_len, int H, int D,
                                                                int64_t a_ld) {
  rb_pdl_launch_dependents();
  extern __shared__ __align__(16) float s_gprep[];
  const int KS = D + 4;                          // row stride: the lanes' 16-byte loads of their own rows spread over the banks
  float* Bs = s_gprep;                           // [32][D + 4]
  float* Qs = Bs + GCH * KS;
  float* Ks = Qs + GCH * KS;
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int D4 = D >> 2;
  rb_pdl_wait();
  const int row0 = chunk_row[chunk], m = chunk_len[chunk];
  for (int i = tid; i < GCH * D4; i += 128) {
    const int j = i / D4, d = (i - j * D4) << 2;
    float4 bb = make_float4(0.f, 0.f, 0.f, 0.f), qq = bb, kk = bb;
    if (j < m) {
      const float* row = rows + (int64_t)(row0 + j) * ld;
      bb = *reinterpret_cast<const float4*>(log_alpha + (int64_t)(row0 + j) * a_ld + h * D + d);
      qq = *reinterpret_cast<const float4*>(row + q_off + h * D + d);
      kk = *reinterpret_cast<const float4*>(row + k_off + h * D + d);
      qq.x *= q_scale; qq.y *= q_scale; qq.z *= q_scale; qq.w *= q_scale;
    }
    *reinterpret_cast<float4*>(Bs + j * KS + d) = bb;
    *reinterpret_cast<float4*>(Qs + j * KS + d) = qq;
    *reinterpret_cast<float4*>(Ks + j * KS + d) = kk;
  }
  __syncthreads();
  for (int d = tid; d < D; d += 128) {           // the running sums, channel by channel
    float run = 0.f;
#pragma unroll 8
    for (int i = 0; i < GCH; ++i) {
      run += Bs[i * KS + d];
      Bs[i * KS + d] = run;
    }
  }
  __syncthreads();
  float* item = scratch + ((int64_t)chunk * H + h) * gla_item_floats(D);
  {
    // thread: column j = lane, rows i = warp + 4 r
    const int j = lane;
    float acc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = 0.f;
    for (int d = 0; d < D; d += 4) {
      const float4 kj = *reinterpret_cast<const float4*>(Ks + j * KS + d);
      const float4 bj = *reinterpret_cast<const float4*>(Bs + j * KS + d);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int i = warp + 4 * r;
        if (j <= i) {
          const float4 qi = *reinterpret_cast<const float4*>(Qs + i * KS + d);
          const float4 bi = *reinterpret_cast<const float4*>(Bs + i * KS + d);
          acc[r] = fmaf(qi.x * kj.x, expf(bi.x - bj.x), acc[r]);
          acc[r] = fmaf(qi.y * kj.y, expf(bi.y - bj.y), acc[r]);
          acc[r] = fmaf(qi.z * kj.z, expf(bi.z - bj.z), acc[r]);
          acc[r] = fmaf(qi.w * kj.w, expf(bi.w - bj.w), acc[r]);
        }
      }
    }
    float* Mo = item + 2 * GCH * D;
#pragma unroll
    for (int r = 0; r < 8; ++r) Mo[(warp + 4 * r) * GCH + j] = acc[r];
  }
  float* Qt = item;
  float* Kt = item + GCH * D;
  float* Eo = item + 2 * GCH * D + GCH * GCH;
  for (int i = tid; i < GCH * D; i += 128) {
    const int j = i / D, d = i - j * D;
    const float b = Bs[j * KS + d], be = Bs[(GCH - 1) * KS + d];
    Qt[i] = Qs[j * KS + d] * expf(b);
    Kt[i] = Ks[j * KS + d] * expf(be - b);
  }
  for (int d = tid; d < D; d += 128) Eo[d] = expf(Bs[(GCH - 1) * KS + d]);
}

// grid (runs, H, tiles of CT value columns), gscan_threads(CT).  A run is a chain of its chunks, so what counts is a chunk's time
// on one SM.  Warps 0 .. CT / 4 - 1 move the memory on, 4 x 4 values a thread that stay in registers and are left in shared memory
// for the others; the other eight make the outputs from what the chunk starts from, beside them.  Shared memory: two buffers of a
// chunk's item (as the first kernel left it) and the tile's values [32][CT], filled a chunk ahead with cp.async; the memory's
// tile S [D][CT] twice: a chunk reads one and writes the other, so that a chunk has one barrier.
// What bounds a chunk is the SM's shared memory (loads of both products, all of them from it), which 16 columns halve; where 32
// leave half of the SMs without a block they are the better ones (1,901 tokens, 8 heads of 128 x 256, so 64 blocks of 32 columns
// or 128 of 16: 188 us with 32, 124 us with 16, which is 2.1 us a chunk).  With more blocks than that the chunk's item, which every
// tile copies whole, would be read twice as often for nothing.
template <int CT>
__global__ void __launch_bounds__(gscan_threads(CT)) gla_chunk_scan_kernel(
    float* o, const float* scratch, const float* rows, int64_t ld, int v_off,
    float* state, const int* seq_first, const int* seq_count,
    const int* run_chunk0, const int* tok_slot, int H, int D, int Dv) {
  rb_pdl_launch_dependents();
  extern __shared__ __align__(16) float s_gscan[];
  constexpr int NT = gscan_threads(CT), SS = gscan_stride(CT), QUADS = CT / 4, KSPLIT = 32 / QUADS, OUT = 16 / KSPLIT;
  const int item_floats = gla_item_floats(D);
  const int per_buf = item_floats + GCH * CT;
  float* Sa = s_gscan + 2 * per_buf;    // [D][SS]: the memory as this chunk finds it
  float* Sb = Sa + D * SS;              // the memory as this chunk leaves it (the two change places after every chunk)
  const int run = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * CT;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool second = warp >= QUADS;    // the outputs
  // outputs: rows 4 (warp - QUADS) + {0..3}, columns 4 ct + {0..3}; the sum over the channels is shared by KSPLIT lanes, and
  // share ks ends up with row mine_row, columns c0 .. c0 + OUT - 1
  const int ks = lane / QUADS, ct = lane % QUADS, r0 = 4 * (warp - QUADS), mine_row = r0 + (ks & 3);
  const int c0 = 4 * ct + (KSPLIT == 8 ? OUT * (ks >> 2) : 0);
  // the memory's step: channels 4 dt + {0..3}, columns 4 cs + {0..3}
  const int cs = tid % QUADS, dt = tid / QUADS;
  rb_pdl_wait();
  const int first = seq_first[run], n = seq_count[run], chunk0 = run_chunk0[run];
  const int slot = tok_slot[first];
  auto copy_chunk = [&](int ci, int buf) {
    const int row0 = first + ci * GCH, m = min(GCH, n - ci * GCH);
    const float* src = scratch + ((int64_t)(chunk0 + ci) * H + h) * item_floats;
    float* dst = s_gscan + (size_t)buf * per_buf;
    for (int i = tid; i < (item_floats >> 2); i += NT) cp_async16(dst + 4 * i, src + 4 * i);
    if (tid < GCH * QUADS) {
      const int j = tid / QUADS, c4 = (tid % QUADS) << 2;
      const bool real = j < m && col0 + c4 < Dv;
      const float* v = real ? rows + (int64_t)(row0 + j) * ld + v_off + h * Dv + col0 + c4 : rows;
      cp_async16_or_zeros(dst + item_floats + j * CT + c4, v, real);
    }
  };
  const int n_chunks = (n + GCH - 1) / GCH;
  copy_chunk(0, 0);
  cp_async_commit();
  float* mine = state + (((int64_t)slot * H + h) * Dv + col0) * D;      // [column][D]
  const bool steps = !second && 4 * dt < D;
  float S[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) S[i][j] = steps && col0 + 4 * cs + j < Dv ? mine[(int64_t)(4 * cs + j) * D + 4 * dt + i] : 0.f;
  if (steps) {
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(Sa + (4 * dt + i) * SS + 4 * cs) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
  }
  for (int ci = 0, buf = 0; ci < n_chunks; ++ci, buf ^= 1) {
    const int row0 = first + ci * GCH, m = min(GCH, n - ci * GCH);
    cp_async_wait<0>();
    __syncthreads();                  // this chunk's copies have landed, the memory the last chunk left is whole, and
                                      // nobody reads the other buffer any more: the one barrier of a chunk
    if (ci + 1 < n_chunks) {
      copy_chunk(ci + 1, buf ^ 1);    // lands while this chunk is multiplied
      cp_async_commit();
    }
    const float* Ss = (ci & 1) ? Sb : Sa;
    float* Sn = (ci & 1) ? Sa : Sb;
    const float* Qt = s_gscan + (size_t)buf * per_buf;
    const float* Kt = Qt + GCH * D;
    const float* Ms = Kt + GCH * D;
    const float* Es = Ms + GCH * GCH;
    const float* Vs = Qt + item_floats;
    if (second) {
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
      const float* A = Qt + r0 * D;
#pragma unroll 2
      for (int d = 4 * ks; d < D; d += 4 * KSPLIT) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(A + i * D + d);
#pragma unroll
        for (int x = 0; x < 4; ++x) b[x] = *reinterpret_cast<const float4*>(Ss + (d + x) * SS + 4 * ct);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float ai[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            acc[i][0] = fmaf(ai[x], b[x].x, acc[i][0]);
            acc[i][1] = fmaf(ai[x], b[x].y, acc[i][1]);
            acc[i][2] = fmaf(ai[x], b[x].z, acc[i][2]);
            acc[i][3] = fmaf(ai[x], b[x].w, acc[i][3]);
          }
        }
      }
      // the lanes' shares: an exchange halves the rows, a second leaves one of them, with eight shares a third halves the columns
      float sum[4], out[OUT];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float k0 = (ks & 1) ? acc[1][j] : acc[0][j], s0 = (ks & 1) ? acc[0][j] : acc[1][j];
        const float k1 = (ks & 1) ? acc[3][j] : acc[2][j], s1 = (ks & 1) ? acc[2][j] : acc[3][j];
        const float v0 = k0 + __shfl_xor_sync(0xffffffffu, s0, QUADS), v1 = k1 + __shfl_xor_sync(0xffffffffu, s1, QUADS);
        sum[j] = ((ks & 2) ? v1 : v0) + __shfl_xor_sync(0xffffffffu, (ks & 2) ? v0 : v1, 2 * QUADS);
      }
      if constexpr (KSPLIT == 8) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float other = __shfl_xor_sync(0xffffffffu, (ks & 4) ? sum[j] : sum[2 + j], 16);
          out[j] = ((ks & 4) ? sum[2 + j] : sum[j]) + other;
        }
      } else {
#pragma unroll
        for (int j = 0; j < OUT; ++j) out[j] = sum[j];
      }
      // M is zero above its diagonal: a loop of fixed length whose loads run ahead
#pragma unroll 4
      for (int j = 0; j < GCH; j += 4) {
        const float4 m4 = *reinterpret_cast<const float4*>(Ms + mine_row * GCH + j);
        const float mj[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          float v[OUT];
          if constexpr (OUT == 4) {
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(Vs + (j + x) * CT + c0);
          } else {
            *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(Vs + (j + x) * CT + c0);
          }
#pragma unroll
          for (int c = 0; c < OUT; ++c) out[c] = fmaf(mj[x], v[c], out[c]);
        }
      }
      if (mine_row < m) {
        float* to = o + ((int64_t)(row0 + mine_row) * H + h) * Dv + col0 + c0;
#pragma unroll
        for (int j = 0; j < OUT; ++j)
          if (col0 + c0 + j < Dv) to[j] = out[j];
      }
    } else if (steps) {
      // S <- diag(e^{B_end}) S + sum_j Kt_j v_j: the chunk's sum from zero, added once, so that a chunk rounds at the memory's size
      // once and not 33 times (600 tokens with long decays: the memory is off by 1.5e-7, 3.5e-7 with every token added to it)
      const float4 e4 = *reinterpret_cast<const float4*>(Es + 4 * dt);
      const float e[4] = {e4.x, e4.y, e4.z, e4.w};
      float add[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) add[i][j] = 0.f;
#pragma unroll 4
      for (int j = 0; j < GCH; ++j) {
        const float4 k4 = *reinterpret_cast<const float4*>(Kt + j * D + 4 * dt);
        const float4 v4 = *reinterpret_cast<const float4*>(Vs + j * CT + 4 * cs);
        const float ki[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          add[i][0] = fmaf(ki[i], v4.x, add[i][0]);
          add[i][1] = fmaf(ki[i], v4.y, add[i][1]);
          add[i][2] = fmaf(ki[i], v4.z, add[i][2]);
          add[i][3] = fmaf(ki[i], v4.w, add[i][3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) S[i][j] = fmaf(e[i], S[i][j], add[i][j]);
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(Sn + (4 * dt + i) * SS + 4 * cs) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
    }
  }
  if (steps) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (col0 + 4 * cs + j < Dv) {
#pragma unroll
        for (int i = 0; i < 4; ++i) mine[(int64_t)(4 * cs + j) * D + 4 * dt + i] = S[i][j];
      }
  }
}

}  // namespace

// alpha [T, C] from rows[t, a_off .. a_off + rank): C = heads x channels outputs of A2 [C, rank] plus bias [C].
// as_log: its logarithm instead (what the chunked kernels add up).
RB_EXPORT int rb_gla_decay(float* alpha, const float* rows, int64_t ld, int a_off, const float* A2, const float* bias, int T,
                           int C, int rank, float tau, int as_log, cudaStream_t stream) {
  if (T == 0) return 0;
  RB_REQUIRE(C > 0 && rank > 0 && tau > 0.f, "rb_gla_decay: bad sizes C=%d rank=%d tau=%g", C, rank, (double)tau);
  RB_REQUIRE((size_t)GLA_DT * rank * sizeof(float) <= 48 * 1024, "rb_gla_decay: a rank of %d is more than a block's shared memory holds", rank);
  int by = (C + 127) / 128;
  if (by > 32) by = 32;
  RB_LAUNCH("gla_decay_kernel", (gla_decay_kernel), dim3((T + GLA_DT - 1) / GLA_DT, by), 128, (size_t)GLA_DT * rank * sizeof(float),
            stream, alpha, rows, ld, a_off, A2, bias, T, C, rank, 1.0f / tau, as_log);
  RB_CHECK_LAUNCH("rb_gla_decay");
  return 0;
}

RB_EXPORT int rb_gla_max_dim() { return 32 * GLA_R; }

// Decays that do not depend on the token (a fixed decay per head, say): after rb_gla_shared_decays() the calling
// thread's next rb_gla_scan or rb_gla_chunked reads ONE row [H * D] of decays (or of their logarithms) for every token.
static thread_local bool t_shared_decays = false;
static bool take_shared_decays() {
  const bool v = t_shared_decays;
  t_shared_decays = false;
  return v;
}
RB_EXPORT int rb_gla_shared_decays() {
  t_shared_decays = true;
  return 0;
}

// o [T, H, Dv] float32.  n_runs runs (seq_first, seq_count; null: every one of the n_runs rows is its own run).
// state: [n_slots, H, Dv, D] float32.
RB_EXPORT int rb_gla_scan(float* o, const float* rows, int64_t ld, int q_off, int k_off, int v_off, const float* alpha,
                          float q_scale, float* state, const int* seq_first, const int* seq_count, const int* tok_slot,
                          int n_runs, int H, int D, int Dv, cudaStream_t stream) {
  const int64_t a_ld = take_shared_decays() ? 0 : (int64_t)H * D;
  if (n_runs == 0) return 0;
  RB_REQUIRE(H > 0 && D > 0 && Dv > 0 && D <= 32 * GLA_R, "rb_gla_scan: bad sizes H=%d D=%d Dv=%d (at most %d key channels)", H,
             D, Dv, 32 * GLA_R);
  int P = 1;
  while (P * GLA_R < D) P *= 2;
#define GO(PP) return launch_scan<PP>(o, rows, ld, q_off, k_off, v_off, alpha, q_scale, state, seq_first, seq_count, tok_slot, n_runs, H, D, Dv, a_ld, stream)
  switch (P) {
    case 1: GO(1);
    case 2: GO(2);
    case 4: GO(4);
    case 8: GO(8);
    case 16: GO(16);
    default: GO(32);
  }
#undef GO
}

// Whether runs of several tokens take the chunked kernels: key sizes that are multiples of 4, up to 128; value sizes
// and row strides that keep every 16-byte copy aligned.
RB_EXPORT int rb_gla_chunked_supports(int D, int Dv, long long ld, int q_off, int k_off, int v_off) {
  return D % 4 == 0 && D > 0 && D <= 128 && Dv > 0 && Dv % 4 == 0 && ld % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0;
}

// Floats of scratch per (chunk, head).
RB_EXPORT long long rb_gla_chunk_floats(int D) { return gla_item_floats(D); }

// The same recurrence for runs of several tokens, in chunks of 32 (see above).  log_alpha [T, H * D]: rb_gla_decay's
// logarithms.  chunk_row, chunk_len: every chunk of every run, the runs' chunks in order; run_chunk0[r]: the first
// chunk of run r.  scratch: n_chunks * H * rb_gla_chunk_floats(D) floats.
RB_EXPORT int rb_gla_chunked(float* o, const float* rows, int64_t ld, int q_off, int k_off, int v_off, const float* log_alpha,
                             float q_scale, float* state, float* scratch, const int* seq_first, const int* seq_count,
                             const int* run_chunk0, const int* chunk_row, const int* chunk_len, const int* tok_slot,
                             int n_runs, int n_chunks, int H, int D, int Dv, cudaStream_t stream) {
  const int64_t a_ld = take_shared_decays() ? 0 : (int64_t)H * D;
  if (n_runs == 0 || n_chunks == 0) return 0;
  RB_REQUIRE(H > 0 && H <= 65535 && rb_gla_chunked_supports(D, Dv, ld, q_off, k_off, v_off) && (uintptr_t)rows % 16 == 0 &&
                 (uintptr_t)scratch % 16 == 0 && (uintptr_t)log_alpha % 16 == 0,
             "rb_gla_chunked: bad sizes H=%d D=%d Dv=%d", H, D, Dv);
  const size_t smem_a = (size_t)(3 * GCH * (D + 4)) * sizeof(float);
  // tiles of 16 columns where those of 32 would leave half of the SMs without a block
  const bool narrow = 2ll * n_runs * H * ((Dv + 31) / 32) <= rb_sm_count();
  const int ct = narrow ? 16 : 32;
  const size_t smem_b = (size_t)(2 * (gla_item_floats(D) + GCH * ct) + 2 * gscan_stride(ct) * D) * sizeof(float);
  static RbOncePerDevice configured;
  if (configured.first()) {
    RB_CUDA(cudaFuncSetAttribute(gla_chunk_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    RB_CUDA(cudaFuncSetAttribute(gla_chunk_scan_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
    RB_CUDA(cudaFuncSetAttribute(gla_chunk_scan_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024));
  }
  RB_REQUIRE(smem_a <= 64 * 1024 && smem_b <= 128 * 1024, "rb_gla_chunked: key size %d needs too much shared memory", D);
  RB_LAUNCH("gla_chunk_prepare_kernel", (gla_chunk_prepare_kernel), dim3(n_chunks, H), 128, smem_a, stream, scratch, rows, ld,
            q_off, k_off, log_alpha, q_scale, chunk_row, chunk_len, H, D, a_ld);
  RB_CHECK_LAUNCH("rb_gla_chunked");
  const dim3 grid(n_runs, H, (Dv + ct - 1) / ct);
  RB_REQUIRE(grid.z <= 65535, "rb_gla_chunked: too many columns");
  if (narrow)
    RB_LAUNCH("gla_chunk_scan_kernel", (gla_chunk_scan_kernel<16>), grid, gscan_threads(16), smem_b, stream, o, scratch, rows, ld,
              v_off, state, seq_first, seq_count, run_chunk0, tok_slot, H, D, Dv);
  else
    RB_LAUNCH("gla_chunk_scan_kernel", (gla_chunk_scan_kernel<32>), grid, gscan_threads(32), smem_b, stream, o, scratch, rows, ld,
              v_off, state, seq_first, seq_count, run_chunk0, tok_slot, H, D, Dv);
  RB_CHECK_LAUNCH("rb_gla_chunked");
  return 0;
}
