// What happens to a product's finished float32 sums before they are stored or added, and the float32 products that are made
// on the tensor cores (gemm_f32_tcgen05.cuh).
#pragma once

#include "rb_common.cuh"

// (null: nothing): bias[n] is added, and the value is multiplied by
// sigmoid(gate[row * ldg + z * gate_batch + n * gate_step]), z the number of the product (a head); a step of
// 0 is one gate for all of a product's values.
struct Tail {
  const float* bias = nullptr;
  const float* gate = nullptr;
  int64_t ldg = 0;
  int64_t gate_batch = 0;
  int gate_step = 1;
};
__device__ __forceinline__ float finished(const Tail& tail, float v, int64_t row, int n, int64_t z) {
  if (tail.bias != nullptr) v += tail.bias[n];
  if (tail.gate != nullptr) v *= 1.0f / (1.0f + expf(-tail.gate[row * tail.ldg + z * tail.gate_batch + n * tail.gate_step]));
  return v;
}

// C[M,N] (+)= alpha * A[M,K] * W[N,K]^T, n_batch times, its operands a fixed distance apart.
struct F32Product {
  float* C; int64_t ldc;
  const float* A; int64_t lda;
  const float* W; int64_t ldw;
  int M, N, K, accumulate;
  float alpha;
  Tail tail;
  int n_batch;
  int64_t batch_c, batch_a, batch_w;
};
// The token tile and the parts of K with which such a product is made, or {0, 0}: it is left to the plain tiles.
struct F32Plan { int bn, parts; };
F32Plan rb_f32_tc_plan(int M, int N, int K, int n_batch, int sms);
int rb_f32_tc(const F32Product& p, F32Plan plan, cudaStream_t stream);
