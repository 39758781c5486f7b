// Incremental decoding: one query token per sequence against a key/value cache.
//
// decode_attention appends the token's key and value to the cache and attends over it in one pass: the caches of a
// step are new tensors one row longer (several continuations may share one past), so every row has to be read and
// written once anyway, and the scores and the weighted sum are taken from the registers that the copy goes through.
// It is bound by that traffic, 8 * (T + 1/2) * dh bytes per head.  A cluster of CTAs shares the keys of one
// (sequence, head); inside a CTA a group of dh / 8 lanes (rounded up to a power of two) owns a key, four keys of a
// group are in flight, and every group keeps its own running maximum, sum and weighted values in fp32.  Groups are
// merged by shuffles, warps through shared memory, CTAs through distributed shared memory, so the kernel needs neither
// a workspace nor a counter that outlives the launch.
// OPT-1.3B (24 layers of 32 heads x 64), 8 sequences of 1000 keys, one token: 15.3 ms -> 3.7 ms a pass together with the GEMM
// below and the native layers, of which the GPU works 2.0; concatenation alone ran at 1 TB/s (6.3 ms) and the fp32 copies of both
// caches took 2.2 ms.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAGuard.h>
#include <cooperative_groups.h>
#include <torch/extension.h>

#include "common.cuh"
#include "gemm_sm100.cuh"

namespace cw {

constexpr int kDecThreads = 256;
constexpr int kDecWarps = kDecThreads / 32;
constexpr int kDecUnroll = 4;            // keys of a lane group in flight

struct DecodeParams {
  const void* qkv;                       // [B, heads, 3 * dh], the token's packed projection
  const void* k_past;                    // [B, heads, T, dh] with the strides below (elements)
  const void* v_past;
  int64_t ks_b, ks_h, ks_t, vs_b, vs_h, vs_t;
  void* k_new;                           // [B, heads, T + 1, dh]
  void* v_new;
  void* out;                             // [B, heads, dh]
  const float* bias;                     // [B, T + 1] or null
  int heads, T, dh;
  float scale;
};

// A partial softmax: maximum, sum of exponentials and weighted values.  An empty part has l == 0 and m == -inf; the
// merge gives it no weight (its factor would be exp(-inf + inf)).
__device__ __forceinline__ float part_weight(float m, float l, float m_all) { return l == 0.f ? 0.f : __expf(m - m_all); }

// LPK lanes share a key, 8 elements each.
template <typename T, int LPK>
__global__ void __launch_bounds__(kDecThreads, 2) decode_attention_kernel(DecodeParams p) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ float s_m[kDecWarps], s_l[kDecWarps];
  __shared__ float s_acc[kDecWarps][LPK * 8];
  __shared__ float c_ml[2];
  __shared__ float c_acc[LPK * 8];

  constexpr int kGroups = 32 / LPK;                      // keys of a warp at a time
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPK, group = lane / LPK;
  const int bh = blockIdx.x / cluster.num_blocks(), b = bh / p.heads, h = bh - b * p.heads;
  const int rank = static_cast<int>(cluster.block_rank()), ranks = static_cast<int>(cluster.num_blocks());
  const int c0 = sub * 8;
  const bool on = c0 < p.dh;

  const T* tok = reinterpret_cast<const T*>(p.qkv) + static_cast<size_t>(bh) * 3 * p.dh;
  const T* kp = reinterpret_cast<const T*>(p.k_past) + b * p.ks_b + h * p.ks_h;
  const T* vp = reinterpret_cast<const T*>(p.v_past) + b * p.vs_b + h * p.vs_h;
  T* kn = reinterpret_cast<T*>(p.k_new) + static_cast<size_t>(bh) * (p.T + 1) * p.dh;
  T* vn = reinterpret_cast<T*>(p.v_new) + static_cast<size_t>(bh) * (p.T + 1) * p.dh;
  const float* bias = p.bias != nullptr ? p.bias + static_cast<size_t>(b) * (p.T + 1) : nullptr;

  float q[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = 0.f;
  if (on) {
    Vec8<T> t;
    t.load(tok + c0);
    t.unpack(q);
  }
  float m = -INFINITY, l = 0.f, acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.f;

  const int keys = p.T + 1;
  constexpr int kStep = kDecWarps * kGroups;             // keys of a CTA between two keys of a group
  // every thread of a warp makes the same number of rounds: the shuffles below need all lanes
  for (int j0 = rank * kStep * kDecUnroll; j0 < keys; j0 += ranks * kStep * kDecUnroll) {
    Vec8<T> kr[kDecUnroll], vr[kDecUnroll];
#pragma unroll
    for (int u = 0; u < kDecUnroll; ++u) {
      const int j = j0 + u * kStep + warp * kGroups + group;
      kr[u].raw = make_uint4(0, 0, 0, 0);
      vr[u].raw = make_uint4(0, 0, 0, 0);
      if (on && j < keys) {
        kr[u].load(j < p.T ? kp + j * p.ks_t + c0 : tok + p.dh + c0);
        vr[u].load(j < p.T ? vp + j * p.vs_t + c0 : tok + 2 * p.dh + c0);
      }
    }
    float s[kDecUnroll];
#pragma unroll
    for (int u = 0; u < kDecUnroll; ++u) {
      const int j = j0 + u * kStep + warp * kGroups + group;
      if (on && j < keys) {
        kr[u].store(kn + static_cast<size_t>(j) * p.dh + c0);
        vr[u].store(vn + static_cast<size_t>(j) * p.dh + c0);
      }
      float f[8];
      kr[u].unpack(f);
      float d = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) d = fmaf(q[i], f[i], d);
#pragma unroll
      for (int o = LPK / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      s[u] = j < keys ? d * p.scale + (bias != nullptr ? __ldg(bias + j) : 0.f) : -INFINITY;
    }
    float mx = m;
#pragma unroll
    for (int u = 0; u < kDecUnroll; ++u) mx = fmaxf(mx, s[u]);
    // until a key with a finite score has been seen the exponentials would be exp(-inf + inf): such keys have no weight
    const float base = mx == -INFINITY ? 0.f : mx;
    const float alpha = __expf(m - base);
    m = mx;
    l *= alpha;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] *= alpha;
#pragma unroll
    for (int u = 0; u < kDecUnroll; ++u) {
      const int j = j0 + u * kStep + warp * kGroups + group;
      if (j < keys) {
        const float e = __expf(s[u] - base);
        l += e;
        float f[8];
        vr[u].unpack(f);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(e, f[i], acc[i]);
      }
    }
  }

  // groups of a warp
#pragma unroll
  for (int o = LPK; o < 32; o <<= 1) {
    const float mo = __shfl_xor_sync(0xffffffffu, m, o), lo = __shfl_xor_sync(0xffffffffu, l, o);
    const float mm = fmaxf(m, mo);
    const float wa = part_weight(m, l, mm), wb = part_weight(mo, lo, mm);
    l = l * wa + lo * wb;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float ao = __shfl_xor_sync(0xffffffffu, acc[i], o);
      acc[i] = acc[i] * wa + ao * wb;
    }
    m = mm;
  }
  if (lane == 0) { s_m[warp] = m; s_l[warp] = l; }
  if (group == 0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) s_acc[warp][c0 + i] = acc[i];
  }
  __syncthreads();
  // warps of the CTA
  if (threadIdx.x < LPK * 8) {
    float mm = s_m[0];
#pragma unroll
    for (int w = 1; w < kDecWarps; ++w) mm = fmaxf(mm, s_m[w]);
    float ll = 0.f, a = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float x = part_weight(s_m[w], s_l[w], mm);
      ll = fmaf(s_l[w], x, ll);
      a = fmaf(s_acc[w][threadIdx.x], x, a);
    }
    c_acc[threadIdx.x] = a;
    if (threadIdx.x == 0) { c_ml[0] = mm; c_ml[1] = ll; }
  }
  cluster.sync();
  // CTAs of the cluster
  if (rank == 0 && static_cast<int>(threadIdx.x) < p.dh) {
    float mm = -INFINITY;
    for (int r = 0; r < ranks; ++r) mm = fmaxf(mm, cluster.map_shared_rank(c_ml, r)[0]);
    float ll = 0.f, a = 0.f;
    for (int r = 0; r < ranks; ++r) {
      const float* ml = cluster.map_shared_rank(c_ml, r);
      const float x = part_weight(ml[0], ml[1], mm);
      ll = fmaf(ml[1], x, ll);
      a = fmaf(cluster.map_shared_rank(c_acc, r)[threadIdx.x], x, a);
    }
    reinterpret_cast<T*>(p.out)[static_cast<size_t>(bh) * p.dh + threadIdx.x] = from_f<T>(a / ll);
  }
  cluster.sync();                        // a CTA's shared memory stays until rank 0 has read it
}

template <typename T, int LPK>
static void launch_decode(const DecodeParams& p, int bh, int ranks, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(bh * ranks);
  cfg.blockDim = dim3(kDecThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  C10_CUDA_CHECK(cudaLaunchKernelEx(&cfg, decode_attention_kernel<T, LPK>, p));
}

template <typename T>
static void dispatch_decode(const DecodeParams& p, int bh, int ranks, cudaStream_t stream) {
  const int lanes = (p.dh + 7) / 8;
  if (lanes <= 4) launch_decode<T, 4>(p, bh, ranks, stream);
  else if (lanes <= 8) launch_decode<T, 8>(p, bh, ranks, stream);
  else if (lanes <= 16) launch_decode<T, 16>(p, bh, ranks, stream);
  else launch_decode<T, 32>(p, bh, ranks, stream);
}

// qkv [B, 1, heads, 3 * dh], caches [B, heads, T, dh] (any strides with dense, 16-byte aligned rows); returns
// (out [B, 1, heads * dh], k [B, heads, T + 1, dh], v).  The caller has checked the forms (ops.decode_ready).
std::vector<torch::Tensor> decode_attention(torch::Tensor qkv, torch::Tensor k_past, torch::Tensor v_past,
                                            c10::optional<torch::Tensor> key_bias, double scale) {
  TORCH_CHECK(qkv.is_cuda() && qkv.is_contiguous() && qkv.dim() == 4 && qkv.size(1) == 1, "decode: qkv must be [B, 1, heads, 3*dh]");
  TORCH_CHECK(k_past.scalar_type() == qkv.scalar_type() && v_past.scalar_type() == qkv.scalar_type() &&
              (qkv.scalar_type() == torch::kBFloat16 || qkv.scalar_type() == torch::kFloat16), "decode: dtypes differ");
  const int64_t B = qkv.size(0), H = qkv.size(2), dh = qkv.size(3) / 3, T = k_past.size(2);
  for (const auto& c : {k_past, v_past}) {
    TORCH_CHECK(c.device() == qkv.device() && c.dim() == 4 && c.size(0) == B && c.size(1) == H && c.size(2) == T && c.size(3) == dh,
                "decode: cache must be [B, heads, T, dh]");
    TORCH_CHECK(c.stride(3) == 1 && c.stride(0) % 8 == 0 && c.stride(1) % 8 == 0 && c.stride(2) % 8 == 0 &&
                reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0, "decode: cache rows must be dense and 16-byte aligned");
  }
  TORCH_CHECK(dh % 8 == 0 && dh >= 8 && dh <= 256 && reinterpret_cast<uintptr_t>(qkv.data_ptr()) % 16 == 0, "decode: head dim");
  TORCH_CHECK(T < (1 << 24) && B * H < (1 << 24), "decode: extents");
  c10::cuda::CUDAGuard guard(qkv.device());
  torch::Tensor bias;
  if (key_bias.has_value()) {
    bias = key_bias->to(torch::kFloat32).contiguous();
    TORCH_CHECK(bias.device() == qkv.device() && bias.dim() == 2 && bias.size(0) == B && bias.size(1) == T + 1,
                "decode: key bias must be [B, T + 1]");
  }
  auto out = torch::empty({B, 1, H * dh}, qkv.options());
  auto k_new = torch::empty({B, H, T + 1, dh}, qkv.options());
  auto v_new = torch::empty({B, H, T + 1, dh}, qkv.options());
  if (B * H == 0) return {out, k_new, v_new};
  DecodeParams p;
  p.qkv = qkv.data_ptr(); p.k_past = k_past.data_ptr(); p.v_past = v_past.data_ptr();
  p.ks_b = k_past.stride(0); p.ks_h = k_past.stride(1); p.ks_t = k_past.stride(2);
  p.vs_b = v_past.stride(0); p.vs_h = v_past.stride(1); p.vs_t = v_past.stride(2);
  p.k_new = k_new.data_ptr(); p.v_new = v_new.data_ptr(); p.out = out.data_ptr();
  p.bias = bias.defined() ? bias.data_ptr<float>() : nullptr;
  p.heads = static_cast<int>(H); p.T = static_cast<int>(T); p.dh = static_cast<int>(dh);
  p.scale = static_cast<float>(scale);
  // CTAs per (sequence, head): as many as are resident at once (two per SM), but not more than there are rounds of keys to
  // share.  A second wave costs more than it balances: start, query load, merge and two cluster barriers are about 8 us of
  // a CTA's life (256 heads x 1001 keys of 64 with four CTAs each: 50 us, with one: 42; the traffic takes 20).
  const int lanes = static_cast<int>((dh + 7) / 8);
  const int lpk = lanes <= 4 ? 4 : (lanes <= 8 ? 8 : (lanes <= 16 ? 16 : 32));
  const int64_t round = static_cast<int64_t>(kDecWarps) * (32 / lpk) * kDecUnroll;
  const int64_t rounds = (T + 1 + round - 1) / round;
  const int64_t room = 2 * at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  int ranks = 1;
  while (ranks < 8 && 2 * ranks * B * H <= room && ranks < rounds) ranks *= 2;
  auto stream = at::cuda::getCurrentCUDAStream();
  if (qkv.scalar_type() == torch::kBFloat16) dispatch_decode<__nv_bfloat16>(p, static_cast<int>(B * H), ranks, stream);
  else dispatch_decode<__half>(p, static_cast<int>(B * H), ranks, stream);
  return {out, k_new, v_new};
}

// ---------------------------------------------------------------------------------------------------------
// y[M, N] = act(x[M, K] W[N, K]^T + b) for a handful of rows (M <= 32): one read of the weights is all the work there
// is.  The persistent tcgen05 kernel has one tile per 256 weight rows (8 CTAs for N = 2048) and cannot ask for enough
// bytes at a time.  Here a warp owns 16 weight rows as the M side of mma.m16n8k16 and the tokens are its N side; the
// warps of a CTA split K between them in chunks of 64 elements and are added up in shared memory (a fixed order).
// The k index of an MMA is summed over, so any bijection of it may be used as long as both operands share it: lane t
// of a quad takes 8 consecutive elements (one 16-byte load) of a row, which are four k pairs of two MMAs.  Weights go
// straight from global memory to registers; nothing is staged.
template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                         uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                  uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

constexpr int kSkChunk = 64;             // k elements of a warp's step: 128 bytes of every weight row

template <typename T, int NT, int W>     // NT groups of 8 tokens, W warps
__global__ void __launch_bounds__(32 * W) skinny_gemm_kernel(const T* __restrict__ x, const T* __restrict__ w,
                                                                    const float* __restrict__ bias,
                                                                    const T* __restrict__ bias16, T* __restrict__ y,
                                                                    T* __restrict__ z, int M, int N, int K, int act) {
  constexpr int U = NT == 1 ? 4 : (NT == 2 ? 2 : 1);        // steps in flight
  __shared__ float red[W][NT * 8][17];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 16;
  const T* w0 = w + static_cast<size_t>(min(n0 + g, N - 1)) * K;           // rows past the end repeat the last one
  const T* w1 = w + static_cast<size_t>(min(n0 + g + 8, N - 1)) * K;
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = warp * kSkChunk; k0 < K; k0 += W * kSkChunk * U) {
    uint4 a[U][2][2], b[U][2][NT];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int k = k0 + u * W * kSkChunk + s * 32 + t * 8;
        const bool ok = k < K;                              // K is a multiple of 8
        a[u][s][0] = ok ? ldg_stream(w0 + k) : make_uint4(0, 0, 0, 0);
        a[u][s][1] = ok ? ldg_stream(w1 + k) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          const int m = i * 8 + g;
          b[u][s][i] = ok && m < M ? __ldg(reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * K + k)) : make_uint4(0, 0, 0, 0);
        }
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          mma_16816<T>(acc[i], a[u][s][0].x, a[u][s][1].x, a[u][s][0].y, a[u][s][1].y, b[u][s][i].x, b[u][s][i].y);
          mma_16816<T>(acc[i], a[u][s][0].z, a[u][s][1].z, a[u][s][0].w, a[u][s][1].w, b[u][s][i].z, b[u][s][i].w);
        }
  }
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    red[warp][i * 8 + 2 * t][g] = acc[i][0];
    red[warp][i * 8 + 2 * t + 1][g] = acc[i][1];
    red[warp][i * 8 + 2 * t][g + 8] = acc[i][2];
    red[warp][i * 8 + 2 * t + 1][g + 8] = acc[i][3];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < NT * 8 * 16; e += 32 * W) {
    const int m = e >> 4, c = e & 15, n = n0 + c;
    if (m >= M || n >= N) continue;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < W; ++q) v += red[q][m][c];
    if (bias != nullptr) v += __ldg(bias + n);
    else if (bias16 != nullptr) v += to_f(bias16[n]);
    const size_t at = static_cast<size_t>(m) * N + n;
    if (z != nullptr) z[at] = from_f<T>(v);
    if (act == kActGelu) v = gelu_fast(v);
    else if (act == kActRelu) v = fmaxf(v, 0.f);
    y[at] = from_f<T>(v);
  }
}

template <typename T>
static void launch_skinny(const GemmArgs& g, cudaStream_t stream) {
  const int grid = (g.N + 15) / 16;
  const T* x = reinterpret_cast<const T*>(g.a);
  const T* w = reinterpret_cast<const T*>(g.b);
  const T* b16 = reinterpret_cast<const T*>(g.bias16);
  T* y = reinterpret_cast<T*>(g.out);
  T* z = reinterpret_cast<T*>(g.z_out);
  // 16 warps share K instead of eight where that does not cost a wave, two CTAs of eight or one of 16 per SM (microseconds with
  // eight and 16): up to one CTA per SM (2304 x 9216, 8 rows 12.9 and 10.6, 16 rows 21.8 and 14.8; 2400 columns 13.3 and 15.8, 22.0
  // and 26.0) and, for few rows and a long K, three (5120 x 8192, 8 rows: 23.8 and 21.9, x 20480: 52.8 and 47.1; 7168: 57.7 and 63.1;
  // 6144 x 2048: 8.5 and 9.2).  With more than 16 rows a warp has one step in flight: up to two CTAs per SM (4736 x 2048, 32
  // rows: 12.4 and 9.2; 8192 x 2048 14.9 and 16.1) and always for a long K (12288 x 8192: 86 and 63).
  const int sms = g.num_sms;
  const bool wide = g.M <= 8    ? grid <= sms || (g.K >= 8192 && grid > 2 * sms && grid <= 3 * sms)
                    : g.M <= 16 ? grid <= sms
                                : grid <= 2 * sms || g.K >= 8192;
#define LAUNCH_SKINNY(NT, W) \
  skinny_gemm_kernel<T, NT, W><<<grid, 32 * W, 0, stream>>>(x, w, g.bias, b16, y, z, g.M, g.N, g.K, g.act)
  if (g.M <= 8) { if (wide) LAUNCH_SKINNY(1, 16); else LAUNCH_SKINNY(1, 8); }
  else if (g.M <= 16) { if (wide) LAUNCH_SKINNY(2, 16); else LAUNCH_SKINNY(2, 8); }
  else { if (wide) LAUNCH_SKINNY(4, 16); else LAUNCH_SKINNY(4, 8); }
#undef LAUNCH_SKINNY
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

void skinny_gemm_launch(const GemmArgs& g, cudaStream_t stream) {
  TORCH_CHECK(g.K % 8 == 0 && ((reinterpret_cast<uintptr_t>(g.a) | reinterpret_cast<uintptr_t>(g.b)) & 15) == 0,
              "GEMM operands must be 16-byte aligned with a row pitch that is a multiple of 8 elements");
  if (g.is_bf16) launch_skinny<__nv_bfloat16>(g, stream);
  else launch_skinny<__half>(g, stream);
}

}  // namespace cw
