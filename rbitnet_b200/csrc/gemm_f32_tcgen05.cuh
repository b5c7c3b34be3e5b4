// float32 products on the tensor cores (included by gemm_tcgen05.cu): C[M,N] (+)= alpha * A[M,K] * W[N,K]^T in 32 bits.
//
// A float32 value is the sum of three bfloat16 values: h = bf16(x), m = bf16(x - h), l = x - h - m, the differences exact
// and l too, for 3 times 8 digits hold all 24 (the method of Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial
// Intelligence Datatype For Higher-Precision Computations", 2019).  A product of two values is then hh + (hm + mh) + (hl + mm + lh) but for
// ml + lm + ll, at most 2^-26 of it, and every product of two parts is exact in the tensor cores' float32.  What they
// lose is in their sums, which are cut off and not rounded, so the large term is summed there over no more than one block of K
// (64 values), into one of two accumulators in tensor memory, and the blocks' sums are added up in registers, rounded.
// The terms of 2^-8 and 2^-16 have an accumulator each for all of K, where the cut is as much smaller.
// Against float64 the result is closer than the FFMA tiles' sums, which round once per value of K (see the figures below).
//
// A sum that is not finite is made again by FFMA (an infinity's parts are infinite and not a number, and a value above the largest
// bfloat16 rounds to infinity), so infinities, NaN and sums near the largest float32 come out as the plain tiles leave them.
// What that costs, us of 600 x 2,048 (2,048 x 2,048 with K 5,632), 66 (342) with finite sums only: 128 tokens with a NaN 73 (636), all
// of them 89 (1,070); 128 tokens with an infinity and no NaN 1,310 (13,700), whose sums are really made again, a thread each.  (All
// sums that are not finite made again, value by value: 128 tokens 4,520 (49,700), all of them 13,400 (98,900); FFMA tiles 145 (1,090).)
// Parts below 2^-133 vanish: values under 2^-110 keep fewer than 24 digits.
//
// A CTA makes a tile of 128 rows of W (the instruction's M side) times BN tokens, or a part of its K.  Sixteen warps fetch float32
// values into registers a block ahead, split them, write the parts into the swizzled operand tiles of one of two stages
// (the planes of a side one below the other, so one instruction reaches two of them: four instructions per 16 values of K) and add up the
// blocks' sums; one thread issues the products.
// What bounds it is shared memory: the products' operands and the splitting's stores and loads take about 3,000 of a block's 3,300 to
// 4,000 cycles, the products' arithmetic 1,536.  2,048 x 11,264 outputs with K 2,048: 680 us, 139 TFLOP/s of float32 (FFMA tiles
// 2,185 us, 43); 2,048 x 4,096 with K 14,336 1,520 (5,500); 600 x 2,048 with K 2,048 69 (146).  Relative error against float64
// (root mean square): K 128 7.5e-8 (FFMA tiles 2.0e-7), 2,048 1.3e-7 (8.1e-7), 14,336 2.1e-7 (1.5e-6).
// (Eight warps of twice the values: 987 us for the first, latencies show; all of an accumulator's products in a row: 766.)
// K in parts: the CTAs of a tile form a cluster, each adds up a share of the token columns from all parts, in order of k.
#pragma once

#include "product_tail.cuh"
#include "rb_tcgen05.cuh"

namespace f32_tc {

constexpr int WARPS = 16, THREADS = WARPS * 32;

template <int BN> constexpr int stage_bytes() { return 3 * (BM + BN) * BK * 2; }

// four neighbours of a row as three planes of bfloat16, 8 bytes each
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void split4(const float4& x, uint2 (&plane)[3]) {
  float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    plane[q].x = pack2(v[0], v[1]);
    plane[q].y = pack2(v[2], v[3]);
    if (q == 2) break;
    v[0] -= __uint_as_float(plane[q].x << 16);
    v[1] -= __uint_as_float(plane[q].x & 0xffff0000u);
    v[2] -= __uint_as_float(plane[q].y << 16);
    v[3] -= __uint_as_float(plane[q].y & 0xffff0000u);
  }
}

template <int BN>
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_kernel(const F32Product p, int n_t_tiles, int parts) {
  constexpr int STEP = 2 * WARPS, W_ROWS = BM / STEP, X_ROWS = BN / STEP;      // rows of a thread, STEP apart
  constexpr int COLS = BN / (WARPS / 4);                                       // token columns of a warp
  constexpr int TMEM_COLS = 4 * BN;                                            // hh of even and odd blocks, 2^-8, 2^-16
  static_assert(TMEM_COLS == 256 || TMEM_COLS == 512, "tensor memory");
  static_assert(BN * BM * 4 <= 2 * stage_bytes<BN>(), "the stages hold a tile's sums");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_bar[2], done_bar[2];
  __shared__ uint32_t tmem_holder;
  rb_pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool issuing = rb_uniform_warp() == 0;
  const int64_t z = blockIdx.z;
  const float* A = p.A + z * p.batch_a;
  const float* W = p.W + z * p.batch_w;
  float* C = p.C + z * p.batch_c;
  const int part = blockIdx.x % parts, tile = blockIdx.x / parts;
  const int n0 = tile / n_t_tiles * BM, t0 = tile % n_t_tiles * BN;
  const int blocks = (p.K + BK - 1) / BK;
  const int b_first = (int)((int64_t)blocks * part / parts), n_blocks = (int)((int64_t)blocks * (part + 1) / parts) - b_first;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&full_bar[s], WARPS);
      mbar_init(&done_bar[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_holder;
  // A sum that is not finite as FFMA leaves it over all of K, in its order; called by whole warps, one token each.  A token with a NaN
  // among its values (what a row looks like once anything in it has overflowed) has no other sums, and is known by one look at the row.
  auto settled = [&](float v, bool in, int m, int n) -> float {
    const bool bad = in && !(fabsf(v) <= 3.402823466e+38f);
    if (!__any_sync(0xffffffffu, bad)) return v;
    const float* a = A + (int64_t)m * p.lda;
    bool nan = false;
    for (int k = lane * 4; k < p.K; k += 128) {
      const float4 x = *reinterpret_cast<const float4*>(a + k);
      nan |= x.x != x.x || x.y != x.y || x.z != x.z || x.w != x.w;
    }
    nan = __any_sync(0xffffffffu, nan);
    if (!bad) return v;
    if (nan) return __uint_as_float(0x7fffffffu);
    const float* w = W + (int64_t)n * p.ldw;
    v = 0.f;
#pragma unroll 4
    for (int k = 0; k < p.K; k += 4) {
      const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
      v = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, v))));
    }
    return v;
  };
  auto value = [&](float v, int m, int n) -> float { return finished(p.tail, p.alpha == 1.0f ? v : v * p.alpha, m, n, z); };

  const int my_row = warp * 2 + (lane >> 4), my_k = (lane & 15) * 4;
  // a row's 128 bytes lie at row * 128, its 16-byte pieces exchanged by the row's number modulo 8 (rows STEP apart: the same)
  const uint32_t my_at = (uint32_t)my_row * 128u + (uint32_t)((((lane & 15) >> 1) ^ (my_row & 7)) << 4) + (uint32_t)((lane & 1) << 3);
  float4 w[W_ROWS], x[X_ROWS];
  // Rows behind the last are the last again (their sums are dropped), values of K behind the last are made zero when they are
  // split: every load is made, so that none is waited for where it is asked for.
  const float* from_w[W_ROWS];
  const float* from_x[X_ROWS];
#pragma unroll
  for (int i = 0; i < W_ROWS; ++i) from_w[i] = W + (int64_t)min(n0 + my_row + STEP * i, p.N - 1) * p.ldw;
#pragma unroll
  for (int i = 0; i < X_ROWS; ++i) from_x[i] = A + (int64_t)min(t0 + my_row + STEP * i, p.M - 1) * p.lda;
  auto k_of = [&](int block) { return min((b_first + min(block, n_blocks - 1)) * BK + my_k, p.K - 4); };
  // a block's values go out of the registers, and the next block's are asked for in their place
  auto put = [&](int block) {
    uint8_t* stage = smem + (block & 1) * stage_bytes<BN>() + my_at;
    const int next = k_of(block + 1);
    if ((b_first + block + 1) * BK > p.K && (b_first + block) * BK + my_k >= p.K) {
#pragma unroll
      for (int i = 0; i < W_ROWS; ++i) w[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < X_ROWS; ++i) x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < W_ROWS; ++i) {
      uint2 plane[3];
      split4(w[i], plane);
      w[i] = *reinterpret_cast<const float4*>(from_w[i] + next);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(stage + (q * BM + i * STEP) * 128) = plane[q];
    }
#pragma unroll
    for (int i = 0; i < X_ROWS; ++i) {
      uint2 plane[3];
      split4(x[i], plane);
      x[i] = *reinterpret_cast<const float4*>(from_x[i] + next);
#pragma unroll
      for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(stage + (3 * BM + q * BN + i * STEP) * 128) = plane[q];
    }
    fence_async_shared();
    tcgen05_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&full_bar[block & 1]);
  };
  bool ok = true;
  // the first warp issues a block's products once all warps have put their rows
  constexpr uint32_t one = make_idesc(BN), two = make_idesc(2 * BN);
  constexpr uint64_t K_STEP = UMMA_K * 2 >> 4;
  const uint64_t first_stage = smem_desc_sw128(smem_u32(smem));
  auto issue = [&](int b) {
    if (!mbar_wait_warp(&full_bar[b & 1], (b >> 1) & 1, 2)) return;        // (noticed by everybody's wait for these products)
    tcgen05_fence_after();
    const uint32_t hh = tmem_base + (uint32_t)((b & 1) * BN), low = tmem_base + 2 * BN;
    const uint64_t w_h = first_stage + (uint64_t)((b & 1) * (stage_bytes<BN>() >> 4)), w_m = w_h + (BM * 128 >> 4), w_l = w_m + (BM * 128 >> 4);
    const uint64_t x_h = w_l + (BM * 128 >> 4), x_m = x_h + (BN * 128 >> 4);
    if (elect_one()) {
#pragma unroll
      for (int k4 = 0; k4 < BK / UMMA_K; ++k4) {
        umma_bf16(hh, w_h + k4 * K_STEP, x_h + k4 * K_STEP, one, k4 > 0 ? 1u : 0u);
        umma_bf16(low, w_h + k4 * K_STEP, x_m + k4 * K_STEP, two, b > 0 || k4 > 0 ? 1u : 0u);      // hm and hl
        umma_bf16(low, w_m + k4 * K_STEP, x_h + k4 * K_STEP, two, 1u);                             // mh and mm
        umma_bf16(low + BN, w_l + k4 * K_STEP, x_h + k4 * K_STEP, one, 1u);                        // lh
      }
      tcgen05_commit(&done_bar[b & 1]);
    }
    __syncwarp();
  };
  const int quarter = warp & 3, c0 = (warp >> 2) * COLS;
  const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
  float sum[COLS];
#pragma unroll
  for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
#pragma unroll
  for (int i = 0; i < W_ROWS; ++i) w[i] = *reinterpret_cast<const float4*>(from_w[i] + k_of(0));      // the weights do not depend on the kernel before
  rb_pdl_wait();
#pragma unroll
  for (int i = 0; i < X_ROWS; ++i) x[i] = *reinterpret_cast<const float4*>(from_x[i] + k_of(0));
  put(0);
  if (issuing) issue(0);
  for (int b = 0; ok && b < n_blocks; ++b) {
    if (b + 1 < n_blocks) {
      put(b + 1);                                         // the products of block b - 1, which read that stage, are done
      if (issuing) issue(b + 1);
    }
    ok = mbar_wait(&done_bar[b & 1], (b >> 1) & 1, 3);
    ok = __all_sync(0xffffffffu, ok);
    tcgen05_fence_after();
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
      uint32_t r[16];
      tmem_ld16(lanes + (uint32_t)((b & 1) * BN + c), r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(r[j]);
    }
  }
#pragma unroll
  for (int c = 0; c < COLS; c += 16) {
    uint32_t r[16], s[16];
    tmem_ld16(lanes + (uint32_t)(2 * BN + c), r);
    tmem_ld16(lanes + (uint32_t)(3 * BN + c), s);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(r[j]) + __uint_as_float(s[j]);
  }
  const int row = quarter * 32 + lane, n = n0 + row;
  if (parts > 1) {
    float* red = reinterpret_cast<float*>(smem);          // [token column][row of W]
#pragma unroll
    for (int j = 0; j < COLS; ++j) red[(c0 + j) * BM + row] = sum[j];
  } else {
    float* dst = C + (int64_t)(t0 + c0) * p.ldc + n;
    const int left = p.M - (t0 + c0);
    const bool in = n < p.N;
#pragma unroll
    for (int c = 0; c < COLS; c += 16) {
      float old[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) old[j] = in && p.accumulate && c + j < left ? dst[(int64_t)(c + j) * p.ldc] : 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (c + j < left) {
          const float v = settled(sum[c + j], in, t0 + c0 + c + j, n);
          if (in) {
            const float done = value(v, t0 + c0 + c + j, n);
            dst[(int64_t)(c + j) * p.ldc] = p.accumulate ? old[j] + done : done;
          }
        }
    }
  }
  if (parts > 1) {
    __syncwarp();
    cluster_sync_all();
    const int my = (int)cluster_rank(), srow = threadIdx.x % BM, sn = n0 + srow;
    const uint32_t red = smem_u32(smem) + (uint32_t)srow * 4;
    const bool in = sn < p.N;
    for (int col = my + parts * (threadIdx.x / BM); col < BN && t0 + col < p.M; col += parts * (THREADS / BM)) {
      float* dst = C + (int64_t)(t0 + col) * p.ldc + sn;
      const float old = in && p.accumulate ? *dst : 0.f;
      float from[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        from[r] = 0.f;
        if (r < parts) {
          uint32_t there;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(red + (uint32_t)(col * BM) * 4), "r"((uint32_t)r));
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(from[r]) : "r"(there));
        }
      }
      float v = from[0];
#pragma unroll
      for (int r = 1; r < 8; ++r) v += from[r];
      v = settled(v, in, t0 + col, sn);
      if (in) {
        v = value(v, t0 + col, sn);
        *dst = p.accumulate ? old + v : v;
      }
    }
    __syncwarp();
    cluster_sync_all();                                   // nobody's shared memory goes away while another rank reads it
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

template <int BN> int launch(const F32Product& p, int parts, cudaStream_t stream) {
  constexpr int smem = 2 * stage_bytes<BN>() + 1024;
  auto kernel = gemm_f32_kernel<BN>;
  static RbOncePerDevice configured;
  if (configured.first()) RB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int64_t n_t = (p.M + BN - 1) / BN, ctas = (p.N + BM - 1) / BM * n_t * parts;
  RB_REQUIRE(ctas <= 0x7fffffff, "rb_gemm_simple: M=%d N=%d: too large for one launch", p.M, p.N);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, 1, p.n_batch);
  cfg.blockDim = dim3(THREADS, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = rb_pdl_enabled() ? 2 : 1;
  RB_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, (int)n_t, parts));
  return 0;
}

}  // namespace f32_tc

// Token tile and parts of K by waves of CTAs, one to an SM (clusters of four leave a tenth of the SMs without one): a block of K
// takes 2.2 us with 128 tokens and 1.75 with 64, a CTA 5 us beside its blocks.  us with 128 tokens in 1, 2, 4 parts and with 64
// in 1, 4: K 2,048: 64 x 2,048 outputs 77, 40, 23, 64, 20; 600 x 2,048 75, 80, 69, 128, 97; 600 x 11,264 223, 246, 321, 387, 516;
// K 14,336, 2,048 x 4,096 1,744, 1,560, 1,832, 2,945, 3,404.  (Eight parts: 22 for the first; clusters of eight fit the chip badly.)
// The plain tiles keep what is too small to fill the SMs and what would be mostly padding (us plain and here): K 192, 300 x 512
// outputs 9.7, 9.8, x 2,048 16.9, 10.8; K 512, 100 x 256 7.0, 8.6, 300 x 256 11.1, 9.0; K 1,024, 300 x 128 9.8, 12.1;
// K 128, 1,000 x 512 9.4, 9.0; 64 products of 4,000 x 64, K 256 214, 247; K below 128 is mostly the blocks' padding
// (70 x 96, K 96: 7.7, 9.1).
F32Plan rb_f32_tc_plan(int M, int N, int K, int n_batch, int sms) {
  const int64_t tiles = (int64_t)((N + 63) / 64) * ((M + 63) / 64) * n_batch;
  const int64_t padded = (int64_t)((N + BM - 1) / BM) * BM;
  if (K < 128 || tiles < 16 || tiles * K < 10240 || (K < 512 ? 2 * padded > 3 * (int64_t)N : padded > 2 * (int64_t)N)) return F32Plan{0, 0};
  const int blocks = (K + BK - 1) / BK;
  F32Plan best{0, 0};
  double least = 0;
  for (int bn = 64; bn <= 128; bn += 64)
    for (int parts = 1; parts <= 4 && parts <= blocks; parts *= 2) {
      const int64_t ctas = (int64_t)((N + BM - 1) / BM) * ((M + bn - 1) / bn) * n_batch * parts, together = parts == 4 ? sms - sms / 9 : sms;
      const double time = (double)((ctas + together - 1) / together) * ((blocks + parts - 1) / parts * (bn == 128 ? 2.2 : 1.75) + 5.0);
      if (best.bn == 0 || time < least) { best = F32Plan{bn, parts}; least = time; }
    }
  return best;
}

// The same for tests: the token tile (0: plain tiles) and the parts of a float32 product whose rows have 16-byte loads.
RB_EXPORT int rb_f32_tc_plan_of(int M, int N, int K, int n_batch, int sms, int* out) {
  const F32Plan plan = rb_f32_tc_plan(M, N, K, n_batch, sms);
  out[0] = plan.bn; out[1] = plan.parts;
  return 0;
}

int rb_f32_tc(const F32Product& p, F32Plan plan, cudaStream_t stream) {
  return plan.bn == 128 ? f32_tc::launch<128>(p, plan.parts, stream) : f32_tc::launch<64>(p, plan.parts, stream);
}
