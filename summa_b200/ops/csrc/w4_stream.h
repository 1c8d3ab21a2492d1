// Launcher of the weight-streaming 4-bit projection (w4_stream.cu) for the C entries in quant.cu and hquant.cu.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sb {

// Epilogue of the qkv projection of a decode step: rotary embedding at the device-side position and
// the append of k / v to the cache, as the separate kernel of `attention_decode.cu` does them.
struct RopeAppend {
  const float* cos_t;      // [max_pos, D/2]; null = plain epilogue
  const float* sin_t;
  __nv_bfloat16* kc;       // caches `[B, cap, Hkv, D]` addressed through the strides below
  __nv_bfloat16* vc;
  const int* pos_ptr;
  int Hq, Hkv, D, cap;
  long c_sb, c_ss, c_sh;
};

enum W4StreamMode { W4S_PLAIN = 0, W4S_GATED = 1, W4S_ROPE = 2 };

struct W4StreamArgs {
  const __nv_bfloat16* x;          // [M, K], row stride ldx (elements, multiple of 8), 16-byte aligned
  const uint32_t* wk8;             // [K / 8, N] repacked codes, 16-byte aligned
  const __nv_bfloat16* scales;     // [K / 128, N], 8-byte aligned
  const __nv_bfloat16* residual;   // [M, N] or null (plain mode)
  __nv_bfloat16* y;                // [M, N]; gated: [M, N / 2]
  int M, N, K;
  long ldx;
  const float* gamma;              // fp32 [K]: y = rmsnorm(x; gamma, eps) @ W; null = no norm
  float eps;
  int static_w;                    // nothing in flight on the stream writes codes or scales: they may be requested early
  RopeAppend rope;                 // W4S_ROPE only
};

constexpr int W4S_MAX_ROWS = 8;
// Whether this kernel is ahead of the tcgen05 one (sb_w4a16_gemm). Up to 8 rows as long as x fits its shared memory in one pass
// (M 8, K 4096, N 28672: 28.7 us, there 39.9 for 12 rows; M 4, K 14336, N 4096: 19.0 us, there 19.6 for 6 rows; otherwise K is
// walked in passes, each with its own staging). From 9 rows on it would need a second set of mma columns.
bool w4_stream_preferred(int M, int K);
int launch_w4_stream(const W4StreamArgs& a, W4StreamMode mode, cudaStream_t st);

}  // namespace sb
