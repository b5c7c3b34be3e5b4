// Plain matrix product on the CUDA cores: C[M,N] (+)= alpha * A[M,K] * W[N,K]^T.
//
// This is the true 32-bit path's product (FFMA with float32 accumulation; of many rows times a K of 128 and more the tensor cores
// make it from values split without loss, see gemm_f32_tcgen05.cuh) and the product for shapes that the
// bfloat16 tensor-core kernel refuses.  W is row-major [out, in], the layout the
// reference indexes as w[i + o*n_in] (crates/bitnet-core/src/llama/model.rs:67-91),
// so no weight is transposed at load.  Every sum is float32 and its order is fixed by the kernel that makes it: tiles of
// outputs add over k in ascending order; a product of few rows adds by lanes (lane l takes every 32nd group of four values)
// and then over the lanes, and the block's warps where they share K, in a fixed tree.
#include "product_tail.cuh"

namespace {

// ---- tiles of outputs
// 64 x 64 outputs a block of 128 threads, 8 x 4 a thread.  What bounds it is the multiply-adds and the shared memory that
// feeds them, so LK values of k are fetched into registers, 16 bytes a load where the rows allow (VEC), while those before them are
// multiplied, and there are two buffers: one barrier per LK, and no warp waits for memory between two of them.  Where the
// tiles are too few to give every SM several, K is cut into 2, 4 or 8 parts whose blocks form a cluster; every block then
// adds up a share of the tile's rows from all parts, in the order of k.
// 2,048 x 11,264 outputs with K 2,048 in 2,215 us (43 TFLOP/s; 2,392 before with tiles of 128 x 128, values loaded one by one
// and no part of K in flight while the one before was multiplied), 647 x 2,048 in 159 (442), 64 x 2,048 in 32 (370).
constexpr int TILE = 64, LK = 16, PITCH = TILE + 4, TILE_THREADS = 128;

// Four finished neighbours of a row.
template <typename TC>
__device__ __forceinline__ void leave4(TC* C, int64_t ldc, int M, int N, int m, int n, float (&v)[4], int accumulate,
                                       float alpha, const Tail& tail) {
  if (m >= M) return;
  TC* p = C + (int64_t)m * ldc + n;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (n + j < N) v[j] = finished(tail, alpha == 1.0f ? v[j] : v[j] * alpha, m, n + j, blockIdx.z);
  if (n + 4 <= N && (uintptr_t)p % (4 * sizeof(TC)) == 0) {
    if (accumulate) {
      float old[4];
      rb_load4(p, old);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] += old[j];
    }
    rb_store4(p, v);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (n + j < N) p[j] = rb_from_float<TC>(accumulate ? v[j] + rb_to_float<TC>(p[j]) : v[j]);
}

template <bool VEC, typename TA, typename TC>
__global__ void __launch_bounds__(TILE_THREADS, 4) gemm_tile_kernel(
    TC* C, int64_t ldc, const TA* A, int64_t lda, const TA* W, int64_t ldw, int M, int N,
    int K, int accumulate, float alpha, Tail tail, int64_t batch_c, int64_t batch_a, int64_t batch_w, int n_parts) {
  constexpr int FETCH = TILE * LK / 4 / TILE_THREADS;      // groups of four values a thread fetches of each operand
  rb_pdl_launch_dependents();
  // blockIdx.z: one of several independent products of equal sizes, their operands a fixed distance apart
  C += blockIdx.z * batch_c;
  A += blockIdx.z * batch_a;
  W += blockIdx.z * batch_w;
  __shared__ __align__(16) float sm[2 * 2 * LK * PITCH];   // [buffer][A, W][LK][PITCH]; at the end [TILE][PITCH], this part's sums
  static_assert(2 * 2 * LK >= TILE, "a tile's sums fit the buffers");
  // blockIdx.x counts parts, tiles of a row of tiles and rows of tiles: y would end at 65,535
  const int part = blockIdx.x % n_parts, tile = blockIdx.x / n_parts, tiles_n = (N + TILE - 1) / TILE;
  const int m0 = tile / tiles_n * TILE, n0 = tile % tiles_n * TILE;
  const int n_blocks = (K + LK - 1) / LK;
  const int k_first = (int)((int64_t)n_blocks * part / n_parts) * LK;
  const int k_end = min(K, (int)((int64_t)n_blocks * (part + 1) / n_parts) * LK);
  // outputs of a thread: rows 4 ty + {0..3} and 32 + 4 ty + {0..3}, columns 4 tx + {0..3}
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float ra[FETCH][4], rw[FETCH][4];
  // A thread's values of a block of K: FETCH groups of four neighbours of a row; for float32 rows without 16-byte loads 4 FETCH
  // values of one k, so that sixteen neighbouring lanes read neighbours and a load of the warp covers two rows and not eight
  // (2,048 x 2,048 with K 130: 46.1 us and 40.7; bfloat16 rows of 1,001 values, 1,024 x 2,048: 169 and 182).
  constexpr bool GROUPS = VEC || sizeof(TA) == 2;
  auto row_in = [&](int i, int j) -> int { return GROUPS ? (threadIdx.x + i * TILE_THREADS) / (LK / 4) : threadIdx.x / LK + (4 * i + j) * (TILE_THREADS / LK); };
  auto k_in = [&](int j) -> int { return GROUPS ? threadIdx.x % (LK / 4) * 4 + j : threadIdx.x % LK; };
  static_assert(TILE_THREADS % LK == 0 && 4 * FETCH * (TILE_THREADS / LK) == TILE, "the values of a block of K are shared out evenly");
  auto fetch = [&](const TA* base, int64_t ld, int at, int rows, int k0, float (&v)[FETCH][4]) {
#pragma unroll
    for (int i = 0; i < FETCH; ++i) {
      v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.f;
      if constexpr (VEC) {                                // K, and so every part's end, is a multiple of four
        if (at + row_in(i, 0) < rows && k0 + k_in(0) < k_end) rb_load4(base + (int64_t)(at + row_in(i, 0)) * ld + k0 + k_in(0), v[i]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (at + row_in(i, j) < rows && k0 + k_in(j) < k_end) v[i][j] = rb_to_float<TA>(base[(int64_t)(at + row_in(i, j)) * ld + k0 + k_in(j)]);
      }
    }
  };
  auto fetch_w = [&](int k0) { fetch(W, ldw, n0, N, k0, rw); };
  auto fetch_a = [&](int k0) { fetch(A, lda, m0, M, k0, ra); };
  auto put = [&](int buf) {
    float* as = sm + buf * 2 * LK * PITCH;
    float* ws = as + LK * PITCH;
#pragma unroll
    for (int i = 0; i < FETCH; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        as[k_in(j) * PITCH + row_in(i, j)] = ra[i][j];
        ws[k_in(j) * PITCH + row_in(i, j)] = rw[i][j];
      }
  };
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  fetch_w(k_first);                                       // the weights do not depend on the kernel before
  rb_pdl_wait();
  fetch_a(k_first);
  put(0);
  __syncthreads();
  for (int k0 = k_first, buf = 0; k0 < k_end; k0 += LK, buf ^= 1) {
    const bool more = k0 + LK < k_end;
    if (more) { fetch_w(k0 + LK); fetch_a(k0 + LK); }
    const float* as = sm + buf * 2 * LK * PITCH + ty * 4;
    const float* ws = sm + buf * 2 * LK * PITCH + LK * PITCH + tx * 4;
#pragma unroll
    for (int kk = 0; kk < LK; ++kk) {
      float a[2][4], w[4];
      rb_load4(as + kk * PITCH, a[0]);
      rb_load4(as + kk * PITCH + 32, a[1]);
      rb_load4(ws + kk * PITCH, w);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i / 4][i % 4], w[j], acc[i][j]);
    }
    if (more) put(buf ^ 1);                               // everybody left that buffer at the last barrier
    __syncthreads();
  }
  if (n_parts == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      leave4(C, ldc, M, N, m0 + i / 4 * 32 + ty * 4 + i % 4, n0 + tx * 4, acc[i], accumulate, alpha, tail);
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) rb_store4(sm + (i / 4 * 32 + ty * 4 + i % 4) * PITCH + tx * 4, acc[i]);
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int rows = TILE / n_parts;
  for (int e = threadIdx.x; e < rows * (TILE / 4); e += TILE_THREADS) {
    const int m = part * rows + e / (TILE / 4), n = e % (TILE / 4) * 4;
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(sm + m * PITCH + n);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    for (int z = 0; z < n_parts; ++z) {
      uint32_t there;
      float4 f;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(at), "r"((uint32_t)z));
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "r"(there));
      v[0] += f.x; v[1] += f.y; v[2] += f.z; v[3] += f.w;
    }
    leave4(C, ldc, M, N, m0 + m, n0 + n, v, accumulate, alpha, tail);
  }
  // nobody leaves while another may still read its sums
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The launch with the parts of a tile as clusters.
template <typename... KArgs, typename... Args>
cudaError_t launch_parts(int n_parts, void (*kernel)(KArgs...), dim3 grid, dim3 block, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = n_parts;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = rb_pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// Parts of K for so many tiles.  K 2,048, us in 1, 2, 4, 8 parts (148 SMs): 32 tiles 98 50 40 30; 224 tiles 220 122 108 109;
// 352 tiles 235 185 164 159; 704 tiles 317 299 302 312; 1,232 tiles 530 497 515 533; 5,632 tiles 2,218 2,215 2,324 2,404:
// many parts even out what the SMs hold while the tiles are few, and cost their exchange once there are enough.
// The exchange costs as much as a block of K.  That is nothing beside a long K, but below 512 it decides: there the parts are those
// with the least of (waves of four blocks an SM, where one that is not full counts 0.4 and 0.6 of its share) x (blocks of K a
// part, and one for the exchange).  K 128: 128 tiles 10.1 10.9 8.9 14.0; 320 tiles 19.3 20.5 20.7 30.6; 1,024 tiles 37.6 43.1
// 51.9 86.8; 2,048 tiles 66 78 98 168.  K 64, 1,024 tiles: 23 30 41 41.
int tile_parts(int64_t tiles, int K, int sms) {
  const int blocks = (K + LK - 1) / LK;
  if (K >= 512) return tiles <= 3 * (int64_t)sms ? 8 : (tiles < 20 * (int64_t)sms ? 2 : 1);
  int best = 1;
  double least = 0;
  for (int p = 1; p <= 8 && p <= blocks; p *= 2) {
    const int64_t all = tiles * p, wave = 4 * (int64_t)sms;
    const double rest = (double)(all % wave) / wave, waves = (double)(all / wave) + (rest > 0 ? 0.4 + 0.6 * rest : 0);
    const double time = waves * ((double)blocks / p + (p > 1 ? 1 : 0));
    if (p == 1 || time < least) { best = p; least = time; }
  }
  return best;
}

// ---- few rows
// A decode step's product is bound by reading W: four outputs a warp for RM (1, 2, 4 or 8) rows, the lanes sharing K, so that a warp
// reads whole lines of W and each value of the rows serves four outputs.  Where the outputs alone do not give every
// scheduler several warps, the block's four warps share the K of four outputs (SHARE) instead of taking four each.  A
// turn's loads of W (16 a lane; 8 with eight rows) are asked for at once, the first turn's before the wait for the kernel before.
// 2,048 x 2,048 (16.8 MB), 1, 3, 8, 16 rows: 4.5, 5.6, 6.5, 10.0 us, where tiles of 64 x 64 took 369 for any of them (32
// blocks, each alone with the whole K); 2,048 x 5,632: 9.3, 12.3, 13.9, 23.3 (996); 11,264 x 2,048: 17, 26, 43, 83 (421);
// 32,000 x 2,048, one row: 42 us, 0.94 of the copy bandwidth.
constexpr int ROW_N = 4, ROW_WARPS = 4;
template <int RM, bool SHARE, bool VEC, typename TA, typename TC>
__global__ void __launch_bounds__(ROW_WARPS * 32) gemm_rows_kernel(
    TC* C, int64_t ldc, const TA* A, int64_t lda, const TA* W, int64_t ldw, int M, int N,
    int K, int accumulate, float alpha, Tail tail, int64_t batch_c, int64_t batch_a, int64_t batch_w) {
  constexpr int V = VEC ? 4 : 1, TURN = RM == 8 ? 2 : 4;
  constexpr int STRIDE = 32 * V * (SHARE ? ROW_WARPS : 1);
  rb_pdl_launch_dependents();
  C += blockIdx.z * batch_c;
  A += blockIdx.z * batch_a;
  W += blockIdx.z * batch_w;
  __shared__ float parts[SHARE ? ROW_WARPS : 1][ROW_N * RM];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (SHARE ? blockIdx.x : blockIdx.x * ROW_WARPS + warp) * ROW_N, m0 = blockIdx.y * RM;
  if (n0 >= N) return;                                  // (SHARE: the whole block)
  const int first = (lane + (SHARE ? 32 * warp : 0)) * V;
  float wv[TURN][ROW_N][V];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < TURN; ++u) {
      const int k = k0 + u * STRIDE;
#pragma unroll
      for (int o = 0; o < ROW_N; ++o) {
        const TA* w = W + (int64_t)(n0 + o) * ldw + k;
        const bool have = k < K && n0 + o < N;
        if constexpr (VEC) {
          if (have) rb_load4(w, wv[u][o]);
          else wv[u][o][0] = wv[u][o][1] = wv[u][o][2] = wv[u][o][3] = 0.f;
        } else {
          wv[u][o][0] = have ? rb_to_float<TA>(*w) : 0.f;
        }
      }
    }
  };
  const TA* a[RM];                                      // rows behind the last are the last again: their sums are dropped
#pragma unroll
  for (int i = 0; i < RM; ++i) a[i] = A + (int64_t)min(m0 + i, M - 1) * lda;
  float acc[ROW_N * RM];
#pragma unroll
  for (int i = 0; i < ROW_N * RM; ++i) acc[i] = 0.f;
  fetch(first);
  rb_pdl_wait();
  for (int k0 = first; k0 < K; k0 += TURN * STRIDE) {
    if (k0 != first) fetch(k0);
#pragma unroll
    for (int u = 0; u < TURN; ++u) {
      const int k = k0 + u * STRIDE;
      if (k < K) {
        float av[RM][V];
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          if constexpr (VEC) rb_load4(a[i] + k, av[i]);
          else av[i][0] = rb_to_float<TA>(a[i][k]);
        }
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int o = 0; o < ROW_N; ++o)
#pragma unroll
            for (int j = 0; j < V; ++j) acc[o * RM + i] = fmaf(av[i][j], wv[u][o][j], acc[o * RM + i]);
      }
    }
  }
  float v;
  if constexpr (ROW_N * RM == 32) {
    v = rb_warp_sum32(acc, lane);
  } else {
    v = 0.f;
#pragma unroll
    for (int i = 0; i < ROW_N * RM; ++i) {
      const float sum = rb_warp_sum(acc[i]);
      if (lane == i) v = sum;
    }
    if (lane >= ROW_N * RM && !SHARE) return;
  }
  if constexpr (SHARE) {
    if (lane < ROW_N * RM) parts[warp][lane] = v;
    __syncthreads();
    if (warp != 0 || lane >= ROW_N * RM) return;
#pragma unroll
    for (int i = 1; i < ROW_WARPS; ++i) v += parts[i][lane];
  }
  const int n = n0 + lane / RM, m = m0 + lane % RM;
  if (n >= N || m >= M) return;
  TC* p = C + (int64_t)m * ldc + n;
  v = finished(tail, alpha == 1.0f ? v : v * alpha, m, n, blockIdx.z);
  if (accumulate) v += rb_to_float<TC>(*p);
  *p = rb_from_float<TC>(v);
}

// Few rows (a decode step) times one matrix per head: a warp makes four outputs of one head for up to eight rows at a
// time, its lanes sharing K, so that the head's matrix is read once, the rows once for four outputs, and heads x N / 16
// blocks are at work instead of a few tiles.  float32 sums (a lane's share in ascending order, then the lanes' shares in a
// fixed tree).  Head h's input values start at column h * head_a of a row.  VEC: four values a load.
constexpr int FEW_ROWS = 8, FEW_OUTS = 4, FEW_WARPS = 4;
template <typename TA, typename TC, bool VEC>
__global__ void __launch_bounds__(FEW_WARPS * 32) per_head_few_rows_kernel(
    TC* C, int64_t ldc, const TA* A, int64_t lda, int head_a, const TA* W, int M, int N,
    int K, Tail tail) {
  rb_pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y, n0 = (blockIdx.x * FEW_WARPS + warp) * FEW_OUTS;
  if (n0 >= N) return;
  const TA* w = W + ((int64_t)h * N + n0) * K;
  const TA* a = A + (int64_t)h * head_a;
  constexpr int V = VEC ? 4 : 1;
  auto fetch = [&](int k, float (&wv)[FEW_OUTS][4]) {
#pragma unroll
    for (int o = 0; o < FEW_OUTS; ++o) {
      const bool have = n0 + o < N && k < K;
      if (VEC) {
        if (have) rb_load4(w + (int64_t)o * K + k, wv[o]);
        else wv[o][0] = wv[o][1] = wv[o][2] = wv[o][3] = 0.f;
      } else {
        wv[o][0] = have ? rb_to_float<TA>(w[(int64_t)o * K + k]) : 0.f;
      }
    }
  };
  float first[FEW_OUTS][4];                              // the matrices do not depend on the kernel before
  fetch(lane * V, first);
  rb_pdl_wait();
  for (int m0 = 0; m0 < M; m0 += FEW_ROWS) {
    float acc[FEW_OUTS * FEW_ROWS];
#pragma unroll
    for (int i = 0; i < FEW_OUTS * FEW_ROWS; ++i) acc[i] = 0.f;
    for (int k = lane * V; k < K; k += 32 * V) {
      float wv[FEW_OUTS][4];
      if (k == lane * V) {
#pragma unroll
        for (int o = 0; o < FEW_OUTS; ++o)
#pragma unroll
          for (int j = 0; j < 4; ++j) wv[o][j] = first[o][j];
      } else {
        fetch(k, wv);
      }
#pragma unroll
      for (int i = 0; i < FEW_ROWS; ++i) {
        if (m0 + i < M) {
          float av[4];
          if (VEC) rb_load4(a + (int64_t)(m0 + i) * lda + k, av);
          else av[0] = rb_to_float<TA>(a[(int64_t)(m0 + i) * lda + k]);
#pragma unroll
          for (int o = 0; o < FEW_OUTS; ++o)
#pragma unroll
            for (int j = 0; j < V; ++j) acc[o * FEW_ROWS + i] = fmaf(av[j], wv[o][j], acc[o * FEW_ROWS + i]);
        }
      }
    }
    const float v = rb_warp_sum32(acc, lane);
    const int n = n0 + lane / FEW_ROWS, m = m0 + lane % FEW_ROWS;
    if (n < N && m < M) C[(int64_t)m * ldc + (int64_t)h * N + n] = rb_from_float<TC>(finished(tail, v, m, n, h));
  }
}

thread_local Tail t_tail;          // of this thread's next call
Tail take_tail() {
  const Tail t = t_tail;
  t_tail = Tail();
  return t;
}

// Few rows by lanes: W is read once for eight of them.  Against tiles, us: 2,048 x 2,048 with 16, 32 rows 10, 17 and 30, 31;
// 11,264 x 2,048 with 16, 20, 32 rows 83, 97, 125 and 86, 87, 87; so more than 16 rows only where the outputs are few.
bool few_rows(int M, int N) { return M <= 16 || (M <= 32 && N <= 4096); }

}  // namespace

// The next rb_gemm_simple, rb_gemm_simple_batched or rb_per_head_few_rows call of this thread adds bias[n] (float32, or
// null) to every finished sum and multiplies it by sigmoid(gate[row * ldg + z * gate_batch + n * gate_step]) (float32, or
// null; z: the number of the product or head).
RB_EXPORT int rb_gemm_simple_next(const float* bias, const float* gate, int64_t ldg, int64_t gate_batch, int gate_step) {
  t_tail.gate_step = gate_step;
  t_tail.bias = bias; t_tail.gate = gate; t_tail.ldg = ldg; t_tail.gate_batch = gate_batch;
  return 0;
}

// C[m, h * N + n] = sum_k A[m, h * head_a + k] * W[h, n, k] for few rows m (any number is right; up to 16 is what it is for).
RB_EXPORT int rb_per_head_few_rows(void* C, int64_t ldc, int c_dtype, const void* A, int64_t lda, int head_a, const void* W,
                                   int a_dtype, int M, int H, int N, int K, cudaStream_t stream) {
  const Tail tail = take_tail();
  if (M == 0 || N == 0 || H == 0) return 0;
  RB_REQUIRE(M > 0 && N > 0 && K > 0 && H > 0 && H <= 65535 && head_a >= K, "rb_per_head_few_rows: bad sizes M=%d H=%d N=%d K=%d (%d apart)",
             M, H, N, K, head_a);
  const dim3 grid((N + FEW_OUTS * FEW_WARPS - 1) / (FEW_OUTS * FEW_WARPS), H);
  const int elem = a_dtype == RB_F32 ? 4 : 2;
  const bool vec = K % 4 == 0 && head_a % 4 == 0 && lda % 4 == 0 && (uintptr_t)A % (4 * elem) == 0 && (uintptr_t)W % (4 * elem) == 0;
#define LAUNCH(TA, TC)                                                                                                  \
  do {                                                                                                                  \
    if (vec) RB_LAUNCH("per_head_few_rows_kernel", (per_head_few_rows_kernel<TA, TC, true>), grid, FEW_WARPS * 32, 0, stream, (TC*)C, ldc, (const TA*)A, lda, head_a, (const TA*)W, M, N, K, tail); \
    else RB_LAUNCH("per_head_few_rows_kernel", (per_head_few_rows_kernel<TA, TC, false>), grid, FEW_WARPS * 32, 0, stream, (TC*)C, ldc, (const TA*)A, lda, head_a, (const TA*)W, M, N, K, tail);    \
  } while (0)
  if (a_dtype == RB_F32 && c_dtype == RB_F32) LAUNCH(float, float);
  else if (a_dtype == RB_BF16 && c_dtype == RB_F32) LAUNCH(__nv_bfloat16, float);
  else if (a_dtype == RB_BF16 && c_dtype == RB_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16);
  else RB_FAIL("rb_per_head_few_rows: unsupported dtypes a=%d c=%d", a_dtype, c_dtype);
#undef LAUNCH
  RB_CHECK_LAUNCH("rb_per_head_few_rows");
  return 0;
}

// Into how many parts plain tiles cut K for this product (1: not; 0: few rows, which are not made by tiles).
RB_EXPORT int rb_gemm_simple_parts(int M, int N, int K, int n_batch) {
  if (few_rows(M, N)) return 0;
  return tile_parts((int64_t)((N + TILE - 1) / TILE) * ((M + TILE - 1) / TILE) * n_batch, K, rb_sm_count());
}

// a_dtype: dtype of A and W; c_dtype: dtype of C.  accumulate: C += instead of C =.
// alpha multiplies the finished sum (1.0 leaves it as it is).
// n_batch products at once: product z reads A + z*batch_a and W + z*batch_w and writes C + z*batch_c
// (distances in elements); block-diagonal matrices are the use.
RB_EXPORT int rb_gemm_simple_batched(void* C, int64_t ldc, int c_dtype, const void* A, int64_t lda, const void* W,
                                     int64_t ldw, int a_dtype, int M, int N, int K, int accumulate, float alpha,
                                     int n_batch, int64_t batch_c, int64_t batch_a, int64_t batch_w,
                                     cudaStream_t stream) {
  const Tail tail = take_tail();
  if (M == 0 || N == 0 || n_batch == 0) return 0;
  RB_REQUIRE(M > 0 && N > 0 && K > 0, "rb_gemm_simple: bad sizes M=%d N=%d K=%d", M, N, K);
  const int elem = a_dtype == RB_F32 ? 4 : 2;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0 &&
                   (uintptr_t)A % (4 * elem) == 0 && (uintptr_t)W % (4 * elem) == 0;
  RB_REQUIRE(n_batch >= 1 && n_batch <= 65535, "rb_gemm_simple: %d products: too many for one launch", n_batch);
#define OF_TYPES(GO)                                                                            \
  do {                                                                                          \
    if (a_dtype == RB_F32 && c_dtype == RB_F32) { if (vec) GO(true, float, float); else GO(false, float, float); }                    \
    else if (a_dtype == RB_BF16 && c_dtype == RB_F32) { if (vec) GO(true, __nv_bfloat16, float); else GO(false, __nv_bfloat16, float); } \
    else if (a_dtype == RB_BF16 && c_dtype == RB_BF16) { if (vec) GO(true, __nv_bfloat16, __nv_bfloat16); else GO(false, __nv_bfloat16, __nv_bfloat16); } \
    else RB_FAIL("rb_gemm_simple: unsupported dtypes a=%d c=%d", a_dtype, c_dtype);             \
  } while (0)
  const int sms = rb_sm_count();
  if (few_rows(M, N)) {
    const int rm = M <= 1 ? 1 : (M <= 2 ? 2 : (M <= 4 ? 4 : 8));
    const int groups = (N + ROW_N - 1) / ROW_N, ys = (M + rm - 1) / rm;
    const bool share = (int64_t)groups * ys * n_batch < (int64_t)sms * 16;
    const dim3 grid(share ? groups : (groups + ROW_WARPS - 1) / ROW_WARPS, ys, n_batch);
#define ROWS(RM, SHARE, VEC, TA, TC) RB_LAUNCH("gemm_rows_kernel", (gemm_rows_kernel<RM, SHARE, VEC, TA, TC>), grid, ROW_WARPS * 32, 0, stream, (TC*)C, ldc, (const TA*)A, lda, (const TA*)W, ldw, M, N, K, accumulate, alpha, tail, batch_c, batch_a, batch_w)
#define GO(VEC, TA, TC)                                                                         \
  do {                                                                                          \
    if (rm == 1) { if (share) ROWS(1, true, VEC, TA, TC); else ROWS(1, false, VEC, TA, TC); }       \
    else if (rm == 2) { if (share) ROWS(2, true, VEC, TA, TC); else ROWS(2, false, VEC, TA, TC); }  \
    else if (rm == 4) { if (share) ROWS(4, true, VEC, TA, TC); else ROWS(4, false, VEC, TA, TC); }  \
    else { if (share) ROWS(8, true, VEC, TA, TC); else ROWS(8, false, VEC, TA, TC); }               \
  } while (0)
    OF_TYPES(GO);
#undef GO
#undef ROWS
  } else {
    const F32Plan plan = a_dtype == RB_F32 && c_dtype == RB_F32 && vec ? rb_f32_tc_plan(M, N, K, n_batch, sms) : F32Plan{0, 0};
    if (plan.bn > 0)
      return rb_f32_tc(F32Product{(float*)C, ldc, (const float*)A, lda, (const float*)W, ldw, M, N, K, accumulate, alpha, tail,
                                  n_batch, batch_c, batch_a, batch_w}, plan, stream);
    const int64_t tiles_n = (N + TILE - 1) / TILE, tiles_m = (M + TILE - 1) / TILE;
    const int parts = tile_parts(tiles_n * tiles_m * n_batch, K, sms);
    RB_REQUIRE(tiles_n * tiles_m * parts <= 0x7fffffff, "rb_gemm_simple: M=%d N=%d: too large for one launch", M, N);
    const dim3 grid((unsigned)(tiles_n * tiles_m * parts), 1, n_batch);
#define GO(VEC, TA, TC)                                                                                                 \
  do {                                                                                                                  \
    const cudaError_t e = launch_parts(parts, gemm_tile_kernel<VEC, TA, TC>, grid, TILE_THREADS, stream, (TC*)C, ldc, (const TA*)A, lda, (const TA*)W, ldw, M, N, K, accumulate, alpha, tail, batch_c, batch_a, batch_w, parts); \
    RB_REQUIRE(e == cudaSuccess, "rb_gemm_simple: launch failed: %s", cudaGetErrorString(e));                           \
  } while (0)
    OF_TYPES(GO);
#undef GO
  }
#undef OF_TYPES
  RB_CHECK_LAUNCH("rb_gemm_simple");
  return 0;
}

RB_EXPORT int rb_gemm_simple(void* C, int64_t ldc, int c_dtype, const void* A, int64_t lda, const void* W,
                             int64_t ldw, int a_dtype, int M, int N, int K, int accumulate,
                             float alpha, cudaStream_t stream) {
  return rb_gemm_simple_batched(C, ldc, c_dtype, A, lda, W, ldw, a_dtype, M, N, K, accumulate, alpha, 1, 0, 0, 0, stream);
}
