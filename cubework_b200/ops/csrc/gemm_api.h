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

// y = act(x W^T + b) for a few rows of x and a 16-bit output goes to the kernel that streams the weights (decode_sm100.cu) up to
// the width from which the tcgen05 tiles keep enough SMs busy.  Microseconds of both, weights from memory, bf16:
//   17 to 32 rows  up to four CTAs of 16 columns per SM (8192 x 2048, 32 rows: 14.9 and 17.5; 6144 x 9216: 45 and 61); what does
//                  not fit in that wave costs a second one (10240 x 2048: 25.5 and 18.0; 50304 x 2048: 75 and 44)
//   9 to 16 rows   up to 16384 columns (16384 x 9216: 62 and 69; 20480 x 5120: 52 and 44), beyond with K around 2048 (50304 x
//                  2048: 46 and 49; x 1024: 28.7 and 27.7; 28672 x 4096: 56 and 45)
//   up to 8 rows   up to 20480 columns (20480 x 9216: 72.5 and 72.7), beyond unless K leaves warps idle (50304 x 768: 24.1 and 21.8)
//                  or is very long (28672 x 9216: 99 and 88); 50304 x 2048: 43 and 49, 20480 x 5120: 44 and 55
constexpr int kSkinnyRows = 32;
inline bool gemm_is_skinny(const GemmArgs& g) {
  if (g.trans_a || !g.trans_b || g.out_f32 || g.M > kSkinnyRows) return false;
  if (g.M > 16) return g.N <= 64 * g.num_sms;
  if (g.M > 8) return g.N <= 16384 || (g.K > 1024 && g.K <= 2048);
  return g.N <= 20480 || (g.K >= 1024 && g.K <= 8192);
}
void skinny_gemm_launch(const GemmArgs& g, cudaStream_t stream);

}  // namespace cw
