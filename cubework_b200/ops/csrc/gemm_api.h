// Host-side interface of the tcgen05 GEMM (no device code: safe to include from plain C++).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cw {

enum Act : int { kActNone = 0, kActGelu = 1, kActRelu = 2 };

struct GemmArgs {
  const void* a;
  const void* b;
  void* out;
  void* z_out = nullptr;
  const float* bias = nullptr;
  const void* bias16 = nullptr;     // bias in the operands' type instead (skinny products only)
  int M, N, K;
  bool trans_a, trans_b;
  bool is_bf16 = true;
  bool out_f32 = false;
  int act = kActNone;
  bool allow_split_k = true;
  int num_sms = 148;
  int* status = nullptr;
};

void gemm_launch(const GemmArgs& g, cudaStream_t stream);

// y = act(x W^T + b) with at most this many rows of x and a 16-bit output (decode_sm100.cu)
constexpr int kSkinnyRows = 32;
void skinny_gemm_launch(const GemmArgs& g, cudaStream_t stream);

}  // namespace cw
