// Launcher of the weight-streaming bf16 projection (bf16_stream.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sb {

struct Bf16StreamArgs {
  const __nv_bfloat16* x;          // [M, K], row stride ldx
  const __nv_bfloat16* w;          // [K, N] row-major, row stride ldw; both 16-byte aligned with strides and K multiples of 8
  const void* bias;                // [N] bf16 or fp32, or null
  int bias_is_bf16;
  const __nv_bfloat16* residual;   // [M, N] contiguous, or null
  __nv_bfloat16* y;                // [M, N], row stride ldy
  int M, N, K;
  long ldx, ldw, ldy;
  const float* gamma;              // fp32 [K]: y = rmsnorm(x; gamma, eps) @ W; null = no norm (needs bf16_stream_one_pass)
  float eps;
};

constexpr int BFS_MAX_ROWS = 8;
bool bf16_stream_takes(const Bf16StreamArgs& a);        // rows, alignment
bool bf16_stream_one_pass(int M, int K);                // the rows of x fit shared memory at once
// `static_w`: the weights were written by nothing that is still in flight, so that they may be requested before the
// preceding kernel has finished (programmatic dependent launch).
int launch_bf16_stream(const Bf16StreamArgs& a, bool static_w, cudaStream_t st);

}  // namespace sb
