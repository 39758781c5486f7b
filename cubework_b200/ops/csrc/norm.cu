// Layer-norm kernels (forward, backward, and the two-pass pieces used when the hidden dimension is
// split over a process group).  One CTA per row, the row held in registers (16-byte loads), statistics in
// fp32.  Backward is persistent over rows so each thread keeps partial dgamma / dbeta for its columns in
// registers; partials are written to a scratch buffer [ctas, H] and summed by a second kernel.
//
// Replaces nn.LayerNorm in LayerNorm1D (cubework/module/parallel_1d/module.py:72-87), the elementwise
// chains of _Layernorm_2D (parallel_2d/_operation.py:307-347 + module.py:142-171) and _Layernorm3D
// (parallel_3d/_operation.py:252-313).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAException.h>
#include <torch/extension.h>

#include "colsum.cuh"
#include "common.cuh"

namespace cw {

constexpr int kNT = 256;
constexpr int kMaxVPT = 8;   // 8 vectors x 8 elements x 256 threads = 16384 columns; kernels are compiled for 1, 2, 3, 4, 8

template <typename T, int VPT>
__device__ __forceinline__ int load_row(const T* row, int H, float (&x)[VPT][8]) {
  int n = 0;
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    const int c = (v * kNT + threadIdx.x) * 8;
    if (c < H) {
      Vec8<T> t;
      t.load(row + c);
      t.unpack(x[v]);
      n = v + 1;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[v][i] = 0.f;
    }
  }
  return n;
}

// 8 consecutive norm parameters as two 16-byte loads (as eight scalar loads, 32 bytes apart between lanes, they kept the
// L1 busier than the rows did: 118 us for 8192 x 5120, which is 168 MB).
__device__ __forceinline__ void load8f(const float* p, float (&f)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
template <typename T>
__device__ __forceinline__ void unpack8(const uint4& raw, float (&f)[8]) {
  const T* h = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = to_f(h[i]);
}
template <typename T>
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 raw;
  T* h = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) h[i] = from_f<T>(f[i]);
  return raw;
}

__device__ __forceinline__ void load8p(const float* p, float (&f)[8]) { load8f(p, f); }
template <typename T>
__device__ __forceinline__ void load8p(const T* p, float (&f)[8]) { unpack8<T>(__ldg(reinterpret_cast<const uint4*>(p)), f); }

// P below: type of the norm parameters, fp32 or that of the rows (models that keep their parameters in 16 bits; converting
// them took two launches per call, as long as the norm of a few rows itself).
//
// MODE 0: local statistics (plain layer norm), optionally of x + res, which is written out as well (HAS_RES).
// MODE 1: statistics supplied (sharded, pass 2).  The row stays in registers as it was loaded (16 bits); the next row
// of the CTA is requested into L2 meanwhile.  8192 x 5120: 118 -> 60 us (168 MB), 73 with the residual (336 MB, which took
// an add of 39 us and a norm of 118).
template <typename T, int MODE, int VPT, bool HAS_RES, typename P>
__global__ void __launch_bounds__(kNT) ln_fwd_kernel(const T* __restrict__ x, const T* __restrict__ res,
                                                     const P* __restrict__ gamma, const P* __restrict__ beta,
                                                     T* __restrict__ sum_out, T* __restrict__ y,
                                                     float* __restrict__ mean_io, float* __restrict__ rstd_io, int rows,
                                                     int H, float eps) {
  __shared__ float red[64];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * H;
    uint4 raw[VPT], rr[HAS_RES ? VPT : 1];
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * kNT + threadIdx.x) * 8;
      raw[v] = c < H ? *reinterpret_cast<const uint4*>(x + base + c) : make_uint4(0, 0, 0, 0);
      if (HAS_RES) rr[v] = c < H ? *reinterpret_cast<const uint4*>(res + base + c) : make_uint4(0, 0, 0, 0);
    }
    // a row that fills the threads once: its parameters are requested with it, not after the two reductions
    float g0[8], be0[8];
    if constexpr (VPT == 1) {
      if (gamma != nullptr && static_cast<int>(threadIdx.x) * 8 < H) {
        load8p(gamma + threadIdx.x * 8, g0);
        load8p(beta + threadIdx.x * 8, be0);
      }
    }
    if (row + gridDim.x < rows) {
      const size_t nbase = base + static_cast<size_t>(gridDim.x) * H;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * kNT + threadIdx.x) * 8;
        if (c < H) {
          prefetch_l2(x + nbase + c);
          if (HAS_RES) prefetch_l2(res + nbase + c);
        }
      }
    }
    if (HAS_RES) {
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * kNT + threadIdx.x) * 8;
        float a[8], b[8];
        unpack8<T>(raw[v], a);
        unpack8<T>(rr[v], b);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] += b[i];
        raw[v] = pack8<T>(a);                         // the normalised value is that of the stored (rounded) sum
        if (c < H) *reinterpret_cast<uint4*>(sum_out + base + c) = raw[v];
      }
    }
    float mean, rstd;
    if (MODE == 0) {
      float s = 0.f, dummy = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        float f[8];
        unpack8<T>(raw[v], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += f[i];
      }
      block_sum2<kNT>(s, dummy, red);
      mean = s / H;
      float q = 0.f;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        if ((v * kNT + threadIdx.x) * 8 < H) {
          float f[8];
          unpack8<T>(raw[v], f);
#pragma unroll
          for (int i = 0; i < 8; ++i) { const float d = f[i] - mean; q += d * d; }
        }
      }
      block_sum2<kNT>(q, dummy, red);
      rstd = rsqrtf(q / H + eps);
      if (threadIdx.x == 0) { mean_io[row] = mean; rstd_io[row] = rstd; }
    } else {
      mean = mean_io[row];
      rstd = rstd_io[row];
    }
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * kNT + threadIdx.x) * 8;
      if (c < H) {
        float f[8];
        unpack8<T>(raw[v], f);
        if (gamma != nullptr) {
          if constexpr (VPT > 1) {
            load8p(gamma + c, g0);
            load8p(beta + c, be0);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = (f[i] - mean) * rstd * g0[i] + be0[i];
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = (f[i] - mean) * rstd;
        }
        *reinterpret_cast<uint4*>(y + base + c) = pack8<T>(f);
      }
    }
  }
}

// Per-row [sum x, sum x^2] for the sharded layer norm (pass 1).
template <typename T, int VPT>
__global__ void __launch_bounds__(kNT) row_moments_kernel(const T* __restrict__ x, float* __restrict__ mom, int rows,
                                                          int H) {
  __shared__ float red[64];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    float xv[VPT][8];
    load_row(x + static_cast<size_t>(row) * H, H, xv);
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int v = 0; v < VPT; ++v)
#pragma unroll
      for (int i = 0; i < 8; ++i) { s += xv[v][i]; q += xv[v][i] * xv[v][i]; }
    block_sum2<kNT>(s, q, red);
    if (threadIdx.x == 0) { mom[2 * row] = s; mom[2 * row + 1] = q; }
  }
}

// Backward.  MODE 0: everything local, optionally plus the gradient that reaches the normalised tensor directly
// (HAS_RES).  MODE 1: only row sums [sum g, sum g*xhat] + parameter partials.  MODE 2: only dx, row sums supplied
// (already reduced over the group) and divided by `hidden`.  Rows stay in registers as they were loaded (16 bits) and
// are converted twice; the next row is requested into L2 meanwhile.  8192 x 5120: 181 -> 83 us, 117 with the residual's
// gradient (336 MB; 205 while it was left at one CTA per SM by its registers).
template <typename T, int MODE, int VPT, bool HAS_RES>
__global__ void __launch_bounds__(kNT, VPT == 1 ? 4 : VPT <= 3 ? 2 : 1) ln_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                     const float* __restrict__ mean, const float* __restrict__ rstd,
                                                     const float* __restrict__ gamma, const T* __restrict__ dres,
                                                     T* __restrict__ dx, float* __restrict__ row_sums,
                                                     float* __restrict__ part_dgamma, float* __restrict__ part_dbeta,
                                                     int rows, int H, float hidden) {
  __shared__ float red[64];
  float dg[VPT][8], db[VPT][8];
#pragma unroll
  for (int v = 0; v < VPT; ++v)
#pragma unroll
    for (int i = 0; i < 8; ++i) { dg[v][i] = 0.f; db[v][i] = 0.f; }

  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * H;
    uint4 xr[VPT], gr[VPT];
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * kNT + threadIdx.x) * 8;
      xr[v] = c < H ? *reinterpret_cast<const uint4*>(x + base + c) : make_uint4(0, 0, 0, 0);
      gr[v] = c < H ? *reinterpret_cast<const uint4*>(dy + base + c) : make_uint4(0, 0, 0, 0);
    }
    {
      const size_t nbase = base + static_cast<size_t>(gridDim.x) * H;
      const bool has_next = row + gridDim.x < rows;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * kNT + threadIdx.x) * 8;
        if (c < H) {
          if (HAS_RES) prefetch_l2(dres + base + c);
          if (has_next) {
            prefetch_l2(x + nbase + c);
            prefetch_l2(dy + nbase + c);
          }
        }
      }
    }
    const float mu = mean[row], rs = rstd[row];
    float s1 = 0.f, s2 = 0.f;
    if (MODE != 2) {
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * kNT + threadIdx.x) * 8;
        if (c < H) {
          float xf[8], gf[8], gm[8];
          unpack8<T>(xr[v], xf);
          unpack8<T>(gr[v], gf);
          if (gamma != nullptr) load8f(gamma + c, gm);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float xhat = (xf[i] - mu) * rs;
            dg[v][i] += gf[i] * xhat;
            db[v][i] += gf[i];
            const float g = gamma != nullptr ? gf[i] * gm[i] : gf[i];
            s1 += g;
            s2 += g * xhat;
          }
        }
      }
      block_sum2<kNT>(s1, s2, red);
      if (MODE == 1 && threadIdx.x == 0) { row_sums[2 * row] = s1; row_sums[2 * row + 1] = s2; }
    } else {
      s1 = row_sums[2 * row];
      s2 = row_sums[2 * row + 1];
    }
    if (MODE != 1) {
      const float m1 = s1 / hidden, m2 = s2 / hidden;
#pragma unroll
      for (int v = 0; v < VPT; ++v) {
        const int c = (v * kNT + threadIdx.x) * 8;
        if (c < H) {
          float xf[8], gf[8], gm[8], rv[8];
          unpack8<T>(xr[v], xf);
          unpack8<T>(gr[v], gf);
          if (gamma != nullptr) load8f(gamma + c, gm);
          if (HAS_RES) unpack8<T>(*reinterpret_cast<const uint4*>(dres + base + c), rv);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float xhat = (xf[i] - mu) * rs;
            const float g = gamma != nullptr ? gf[i] * gm[i] : gf[i];
            xf[i] = (g - m1 - xhat * m2) * rs;
            if (HAS_RES) xf[i] += rv[i];
          }
          *reinterpret_cast<uint4*>(dx + base + c) = pack8<T>(xf);
        }
      }
    }
  }
  if (MODE != 2) {
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      const int c = (v * kNT + threadIdx.x) * 8;
      if (c < H) {
        float4* pg = reinterpret_cast<float4*>(part_dgamma + static_cast<size_t>(blockIdx.x) * H + c);
        float4* pb = reinterpret_cast<float4*>(part_dbeta + static_cast<size_t>(blockIdx.x) * H + c);
        pg[0] = make_float4(dg[v][0], dg[v][1], dg[v][2], dg[v][3]);
        pg[1] = make_float4(dg[v][4], dg[v][5], dg[v][6], dg[v][7]);
        pb[0] = make_float4(db[v][0], db[v][1], db[v][2], db[v][3]);
        pb[1] = make_float4(db[v][4], db[v][5], db[v][6], db[v][7]);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// Warp-per-row layer norm for hidden sizes up to 2048 (backward: up to 1280): a row lives in one warp's registers (NV 16-byte vectors
// per lane), the two statistics are warp shuffles, and nothing synchronises the CTA, so eight rows per CTA are in
// flight with all their loads outstanding.  Optionally fused with the residual add in front of the norm
// (reference: `x = x + dropout(...)` followed by `norm(x)`, benchmark/gpt2/gpt2.py:179-186): forward writes the sum
// and its normalised value, backward adds the gradient that reaches the sum directly.
constexpr int kWarpRows = 8;                 // warps (rows in flight) per CTA
// The backward of rows above 1280 columns takes a CTA per row, four per SM, with the parameter gradients in registers: by
// warps, sixteen rows per SM wait for their loads (32768 x 1600 with a residual 163 us, 120 by CTAs; 4096 x 2048 56 and 32;
// at 1280 65 and 60, without a residual 52 and 54; at 768 99 and 136).
constexpr int kWarpMaxBwd = 1280;

template <typename T, int NV, bool HAS_RES, typename P>
__global__ void __launch_bounds__(32 * kWarpRows)
ln_fwd_warp_kernel(const T* __restrict__ x, const T* __restrict__ res, const P* __restrict__ gamma,
                   const P* __restrict__ beta, T* __restrict__ sum_out, T* __restrict__ y, float* __restrict__ mean_o,
                   float* __restrict__ rstd_o, int rows, int H, float eps) {
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * kWarpRows + (threadIdx.x >> 5);
  const int nwarps = gridDim.x * kWarpRows;
  const float inv_h = 1.0f / H;
  for (int row = warp; row < rows; row += nwarps) {
    const size_t base = static_cast<size_t>(row) * H;
    uint4 raw[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = (v * 32 + lane) * 8;
      raw[v] = c < H ? *reinterpret_cast<const uint4*>(x + base + c) : make_uint4(0, 0, 0, 0);
    }
    // the next row of this warp goes to L2 while this one is processed (costs no registers)
    if (row + nwarps < rows) {
      const size_t nbase = static_cast<size_t>(row + nwarps) * H;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int c = (v * 32 + lane) * 8;
        if (c < H) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(x + nbase + c));
          if (HAS_RES) asm volatile("prefetch.global.L2 [%0];" ::"l"(res + nbase + c));
        }
      }
    }
    if (HAS_RES) {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int c = (v * 32 + lane) * 8;
        if (c < H) {
          const uint4 r = *reinterpret_cast<const uint4*>(res + base + c);
          float a[8], b[8];
          unpack8<T>(raw[v], a);
          unpack8<T>(r, b);
#pragma unroll
          for (int i = 0; i < 8; ++i) a[i] += b[i];
          raw[v] = pack8<T>(a);                       // the normalised value is that of the stored (rounded) sum
          *reinterpret_cast<uint4*>(sum_out + base + c) = raw[v];
        }
      }
    }
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      float f[8];
      unpack8<T>(raw[v], f);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += f[i];
    }
    const float mean = warp_sum(s) * inv_h;
    float q = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      if ((v * 32 + lane) * 8 < H) {
        float f[8];
        unpack8<T>(raw[v], f);
#pragma unroll
        for (int i = 0; i < 8; ++i) { const float d = f[i] - mean; q += d * d; }
      }
    }
    const float rstd = rsqrtf(warp_sum(q) * inv_h + eps);
    if (lane == 0) { mean_o[row] = mean; rstd_o[row] = rstd; }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = (v * 32 + lane) * 8;
      if (c < H) {
        float f[8];
        unpack8<T>(raw[v], f);
        float gg[8], bb[8];
        load8p(gamma + c, gg);
        load8p(beta + c, bb);
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = (f[i] - mean) * rstd * gg[i] + bb[i];
        *reinterpret_cast<uint4*>(y + base + c) = pack8<T>(f);
      }
    }
  }
}

// Backward of the above, for rows of up to kWarpMaxBwd columns.  Each warp keeps the dgamma / dbeta partial sums of its rows
// in a shared-memory strip of its own (in registers they would take 2 * H / 32 per thread, 80 at H = 1280, and hold the kernel
// at eight warps per SM, where it is bound by latency); the warps of a CTA are added up at the end and the CTA writes one
// partial row (summed by colsum_kernel).
template <typename T, int NV, bool HAS_RES>
__global__ void __launch_bounds__(32 * kWarpRows, 2)
ln_bwd_warp_kernel(const T* __restrict__ dy, const T* __restrict__ x, const float* __restrict__ mean,
                   const float* __restrict__ rstd, const float* __restrict__ gamma, const T* __restrict__ dres,
                   T* __restrict__ dx, float* __restrict__ part_dgamma, float* __restrict__ part_dbeta, int rows, int H) {
  extern __shared__ __align__(16) float sacc[];            // [kWarpRows][2][H]
  const int lane = threadIdx.x & 31;
  const int warp = blockIdx.x * kWarpRows + (threadIdx.x >> 5);
  const int nwarps = gridDim.x * kWarpRows;
  const float inv_h = 1.0f / H;
  float* wdg = sacc + static_cast<size_t>(threadIdx.x >> 5) * 2 * H;
  float* wdb = wdg + H;
  for (int i = lane * 4; i < 2 * H; i += 128) *reinterpret_cast<float4*>(wdg + i) = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();

  for (int row = warp; row < rows; row += nwarps) {
    const size_t base = static_cast<size_t>(row) * H;
    uint4 xr[NV], gr[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = (v * 32 + lane) * 8;
      const bool ok = c < H;
      xr[v] = ok ? *reinterpret_cast<const uint4*>(x + base + c) : make_uint4(0, 0, 0, 0);
      gr[v] = ok ? *reinterpret_cast<const uint4*>(dy + base + c) : make_uint4(0, 0, 0, 0);
    }
    // requests that cost no registers: this row's residual gradient (read in the second pass) and the next row's
    // operands go to L2 while the first pass runs
    {
      const size_t nbase = static_cast<size_t>(row + nwarps) * H;
      const bool has_next = row + nwarps < rows;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        const int c = (v * 32 + lane) * 8;
        if (c < H) {
          if (HAS_RES) asm volatile("prefetch.global.L2 [%0];" ::"l"(dres + base + c));
          if (has_next) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(x + nbase + c));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(dy + nbase + c));
          }
        }
      }
    }
    const float mu = mean[row], rs = rstd[row];
    const float nmr = -mu * rs;
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = (v * 32 + lane) * 8;
      if (c < H) {
        float xf[8], df[8];
        unpack8<T>(xr[v], xf);
        unpack8<T>(gr[v], df);
        const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + c)), g1 = __ldg(reinterpret_cast<const float4*>(gamma + c + 4));
        const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        float4* pg = reinterpret_cast<float4*>(wdg + c);
        float4* pb = reinterpret_cast<float4*>(wdb + c);
        float4 a0 = pg[0], a1 = pg[1], b0 = pb[0], b1 = pb[1];
        float ag[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        float ab[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float xhat = fmaf(xf[i], rs, nmr);
          ag[i] = fmaf(df[i], xhat, ag[i]);
          ab[i] += df[i];
          const float g = df[i] * gg[i];
          s1 += g;
          s2 = fmaf(g, xhat, s2);
        }
        pg[0] = make_float4(ag[0], ag[1], ag[2], ag[3]);
        pg[1] = make_float4(ag[4], ag[5], ag[6], ag[7]);
        pb[0] = make_float4(ab[0], ab[1], ab[2], ab[3]);
        pb[1] = make_float4(ab[4], ab[5], ab[6], ab[7]);
      }
    }
    const float m1 = warp_sum(s1) * inv_h, m2 = warp_sum(s2) * inv_h;
    // dx = rs * (dy * gamma - m1 - xhat * m2) = dy * (rs * gamma) + x * kx + k0
    const float kx = -rs * rs * m2, k0 = rs * (mu * rs * m2 - m1);
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = (v * 32 + lane) * 8;
      if (c < H) {
        float xf[8], df[8], o[8];
        unpack8<T>(xr[v], xf);
        unpack8<T>(gr[v], df);
        const float4 g0 = __ldg(reinterpret_cast<const float4*>(gamma + c)), g1 = __ldg(reinterpret_cast<const float4*>(gamma + c + 4));
        const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = fmaf(df[i], rs * gg[i], fmaf(xf[i], kx, k0));
        if (HAS_RES) {
          float rf[8];
          unpack8<T>(*reinterpret_cast<const uint4*>(dres + base + c), rf);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[i] += rf[i];
        }
        *reinterpret_cast<uint4*>(dx + base + c) = pack8<T>(o);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int w = 0; w < kWarpRows; ++w) {
      a += sacc[static_cast<size_t>(w) * 2 * H + i];
      b += sacc[static_cast<size_t>(w) * 2 * H + H + i];
    }
    part_dgamma[static_cast<size_t>(blockIdx.x) * H + i] = a;
    part_dbeta[static_cast<size_t>(blockIdx.x) * H + i] = b;
  }
}

template <typename T, int NV, bool HAS_RES>
static void launch_ln_bwd_warp(int grid, size_t smem, cudaStream_t stream, const void* dy, const void* x, const float* mean,
                               const float* rstd, const float* gamma, const void* dres, void* dx, float* pdg, float* pdb,
                               int rows, int H) {
  auto kern = ln_bwd_warp_kernel<T, NV, HAS_RES>;
  static bool done = false;
  if (!done) {
    C10_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWarpRows * 2 * kWarpMaxBwd * 4));
    done = true;
  }
  kern<<<grid, 32 * kWarpRows, smem, stream>>>(reinterpret_cast<const T*>(dy), reinterpret_cast<const T*>(x), mean, rstd, gamma,
                                               reinterpret_cast<const T*>(dres), reinterpret_cast<T*>(dx), pdg, pdb, rows, H);
}

// ---------------------------------------------------------------------------------------- host side
static void check_rows(const torch::Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous(), "expected a contiguous 2-D CUDA tensor");
  TORCH_CHECK(x.size(1) % 8 == 0 && x.size(1) <= kNT * 8 * kMaxVPT, "hidden size must be a multiple of 8 and <= 16384");
  TORCH_CHECK(x.scalar_type() == torch::kBFloat16 || x.scalar_type() == torch::kFloat16, "expected bf16 / fp16");
}
static int row_grid(int rows) {
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  return std::max(1, std::min(rows, sms * 8));
}
static const float* fptr(const c10::optional<torch::Tensor>& t) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->scalar_type() == torch::kFloat32 && t->is_contiguous(), "norm parameters must be contiguous fp32");
  return t->data_ptr<float>();
}

#define DISPATCH_VPT(H, ...)                                        \
  {                                                                 \
    const int need_ = ((H) / 8 + kNT - 1) / kNT;                    \
    if (need_ <= 1) { constexpr int VPT = 1; __VA_ARGS__ }          \
    else if (need_ <= 2) { constexpr int VPT = 2; __VA_ARGS__ }     \
    else if (need_ <= 3) { constexpr int VPT = 3; __VA_ARGS__ }     \
    else if (need_ <= 4) { constexpr int VPT = 4; __VA_ARGS__ }     \
    else { constexpr int VPT = 8; __VA_ARGS__ }                     \
  }
#define DISPATCH_16(x, ...)                                         \
  if ((x).scalar_type() == torch::kBFloat16) {                      \
    using T = __nv_bfloat16;                                        \
    DISPATCH_VPT((x).size(1), __VA_ARGS__)                          \
  } else {                                                          \
    using T = __half;                                               \
    DISPATCH_VPT((x).size(1), __VA_ARGS__)                          \
  }

// The kernels read norm parameters in 16-byte pieces; a view that starts elsewhere (a slice of a flat buffer) is copied.
static torch::Tensor aligned16(const torch::Tensor& t) {
  return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 ? t : t.clone();
}
static c10::optional<torch::Tensor> aligned16(const c10::optional<torch::Tensor>& t) {
  if (!t.has_value() || !t->defined()) return t;
  return aligned16(*t);
}

static std::vector<torch::Tensor> layer_norm_fwd_cta(torch::Tensor x, const torch::Tensor* res, torch::Tensor gamma,
                                                     torch::Tensor beta, double eps) {
  check_rows(x);
  const int rows = x.size(0), H = x.size(1);
  gamma = aligned16(gamma);
  beta = aligned16(beta);
  auto y = torch::empty_like(x);
  auto mean = torch::empty({rows}, x.options().dtype(torch::kFloat32));
  auto rstd = torch::empty({rows}, x.options().dtype(torch::kFloat32));
  torch::Tensor sum;
  if (res != nullptr) sum = torch::empty_like(x);
  if (rows == 0) return {y, mean, rstd, sum};
  auto stream = at::cuda::getCurrentCUDAStream();
#define LAUNCH_LN_CTA(RES, P)                                                                                             \
  ln_fwd_kernel<T, 0, VPT, RES, P><<<row_grid(rows), kNT, 0, stream>>>(                                                   \
      reinterpret_cast<const T*>(x.data_ptr()), RES ? reinterpret_cast<const T*>(res->data_ptr()) : nullptr,              \
      reinterpret_cast<const P*>(gamma.data_ptr()), reinterpret_cast<const P*>(beta.data_ptr()),                          \
      RES ? reinterpret_cast<T*>(sum.data_ptr()) : nullptr, reinterpret_cast<T*>(y.data_ptr()), mean.data_ptr<float>(),   \
      rstd.data_ptr<float>(), rows, H, static_cast<float>(eps))
  const bool f32 = gamma.scalar_type() == torch::kFloat32;
  DISPATCH_16(x, {
    if (res != nullptr) { if (f32) LAUNCH_LN_CTA(true, float); else LAUNCH_LN_CTA(true, T); }
    else { if (f32) LAUNCH_LN_CTA(false, float); else LAUNCH_LN_CTA(false, T); }
  })
#undef LAUNCH_LN_CTA
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {y, mean, rstd, sum};
}

std::vector<torch::Tensor> layer_norm_fwd(torch::Tensor x, torch::Tensor gamma, torch::Tensor beta, double eps) {
  TORCH_CHECK(gamma.scalar_type() == torch::kFloat32 && beta.scalar_type() == torch::kFloat32 && gamma.is_contiguous() &&
              beta.is_contiguous(), "norm parameters must be contiguous fp32");
  auto r = layer_norm_fwd_cta(x, nullptr, gamma, beta, eps);
  r.pop_back();
  return r;
}

torch::Tensor norm_apply(torch::Tensor x, torch::Tensor mean, torch::Tensor rstd, c10::optional<torch::Tensor> gamma,
                         c10::optional<torch::Tensor> beta) {
  check_rows(x);
  const int rows = x.size(0), H = x.size(1);
  auto y = torch::empty_like(x);
  if (rows == 0) return y;
  auto stream = at::cuda::getCurrentCUDAStream();
  gamma = aligned16(gamma);
  beta = aligned16(beta);
  DISPATCH_16(x, ln_fwd_kernel<T, 1, VPT, false, float><<<row_grid(rows), kNT, 0, stream>>>(
                     reinterpret_cast<const T*>(x.data_ptr()), nullptr, fptr(gamma), fptr(beta), nullptr,
                     reinterpret_cast<T*>(y.data_ptr()), mean.data_ptr<float>(), rstd.data_ptr<float>(), rows, H, 0.f);)
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return y;
}

torch::Tensor row_moments(torch::Tensor x) {
  check_rows(x);
  const int rows = x.size(0), H = x.size(1);
  auto mom = torch::empty({rows, 2}, x.options().dtype(torch::kFloat32));
  if (rows == 0) return mom;
  auto stream = at::cuda::getCurrentCUDAStream();
  DISPATCH_16(x, row_moments_kernel<T, VPT><<<row_grid(rows), kNT, 0, stream>>>(reinterpret_cast<const T*>(x.data_ptr()),
                                                                             mom.data_ptr<float>(), rows, H);)
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return mom;
}

// Launches the backward kernel on caller-provided scratch: part_dgamma / part_dbeta are [grid, H] fp32.
template <int MODE>
static void ln_bwd_launch(const torch::Tensor& dy, const torch::Tensor& x, const float* mean, const float* rstd,
                          const float* gamma, const void* dres, void* dx, float* row_sums, float* pdg, float* pdb, int grid,
                          float hidden, cudaStream_t stream) {
  const int rows = x.size(0), H = x.size(1);
  if (MODE == 0 && dres != nullptr) {
    DISPATCH_16(x, ln_bwd_kernel<T, 0, VPT, true><<<grid, kNT, 0, stream>>>(
                       reinterpret_cast<const T*>(dy.data_ptr()), reinterpret_cast<const T*>(x.data_ptr()), mean, rstd, gamma,
                       reinterpret_cast<const T*>(dres), reinterpret_cast<T*>(dx), row_sums, pdg, pdb, rows, H, hidden);)
  } else {
    DISPATCH_16(x, ln_bwd_kernel<T, MODE, VPT, false><<<grid, kNT, 0, stream>>>(
                       reinterpret_cast<const T*>(dy.data_ptr()), reinterpret_cast<const T*>(x.data_ptr()), mean, rstd, gamma,
                       nullptr, reinterpret_cast<T*>(dx), row_sums, pdg, pdb, rows, H, hidden);)
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
}

// persistent over rows: as many CTAs as are resident at once
static int bwd_grid(int rows, int H) {
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  return std::max(1, std::min(rows, sms * (H <= kNT * 8 ? 4 : 2)));
}

static std::vector<torch::Tensor> layer_norm_bwd_cta(torch::Tensor dy, torch::Tensor x, torch::Tensor mean, torch::Tensor rstd,
                                                     torch::Tensor gamma, const torch::Tensor* dres) {
  check_rows(x);
  check_rows(dy);
  const int rows = x.size(0), H = x.size(1);
  gamma = aligned16(gamma);
  auto dx = torch::empty_like(x);
  auto f32 = x.options().dtype(torch::kFloat32);
  if (rows == 0) return {dx, torch::zeros({H}, f32), torch::zeros({H}, f32)};
  auto dgamma = torch::empty({H}, f32), dbeta = torch::empty({H}, f32);
  const int grid = bwd_grid(rows, H);
  auto scratch = torch::empty({2, grid, H}, f32);
  auto stream = at::cuda::getCurrentCUDAStream();
  float* pdg = scratch.data_ptr<float>();
  float* pdb = pdg + static_cast<size_t>(grid) * H;
  ln_bwd_launch<0>(dy, x, mean.data_ptr<float>(), rstd.data_ptr<float>(), fptr(gamma),
                   dres != nullptr ? dres->data_ptr() : nullptr, dx.data_ptr(), nullptr, pdg, pdb, grid,
                   static_cast<float>(H), stream);
  colsum_launch(pdg, pdb, dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), grid, H, stream);
  return {dx, dgamma, dbeta};
}

std::vector<torch::Tensor> layer_norm_bwd(torch::Tensor dy, torch::Tensor x, torch::Tensor mean, torch::Tensor rstd,
                                          torch::Tensor gamma) {
  return layer_norm_bwd_cta(dy, x, mean, rstd, gamma, nullptr);
}

std::vector<torch::Tensor> norm_bwd_partials(torch::Tensor dy, torch::Tensor x, torch::Tensor mean, torch::Tensor rstd,
                                             c10::optional<torch::Tensor> gamma) {
  check_rows(x);
  check_rows(dy);
  const int rows = x.size(0), H = x.size(1);
  auto f32 = x.options().dtype(torch::kFloat32);
  auto sums = torch::empty({rows, 2}, f32);
  if (rows == 0) return {sums, torch::zeros({H}, f32), torch::zeros({H}, f32)};
  gamma = aligned16(gamma);
  auto dgamma = torch::empty({H}, f32), dbeta = torch::empty({H}, f32);
  const int grid = bwd_grid(rows, H);
  auto scratch = torch::empty({2, grid, H}, f32);
  auto stream = at::cuda::getCurrentCUDAStream();
  float* pdg = scratch.data_ptr<float>();
  float* pdb = pdg + static_cast<size_t>(grid) * H;
  ln_bwd_launch<1>(dy, x, mean.data_ptr<float>(), rstd.data_ptr<float>(), fptr(gamma), nullptr, nullptr, sums.data_ptr<float>(), pdg,
                   pdb, grid, 1.f, stream);
  colsum_launch(pdg, pdb, dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), grid, H, stream);
  return {sums, dgamma, dbeta};
}

torch::Tensor norm_bwd_apply(torch::Tensor dy, torch::Tensor x, torch::Tensor mean, torch::Tensor rstd,
                             c10::optional<torch::Tensor> gamma, torch::Tensor sums, double hidden) {
  check_rows(x);
  check_rows(dy);
  TORCH_CHECK(sums.scalar_type() == torch::kFloat32 && sums.is_contiguous());
  const int rows = x.size(0);
  auto dx = torch::empty_like(x);
  if (rows == 0) return dx;
  auto stream = at::cuda::getCurrentCUDAStream();
  gamma = aligned16(gamma);
  ln_bwd_launch<2>(dy, x, mean.data_ptr<float>(), rstd.data_ptr<float>(), fptr(gamma), nullptr, dx.data_ptr(), sums.data_ptr<float>(),
                   nullptr, nullptr, row_grid(rows), static_cast<float>(hidden), stream);
  return dx;
}

// ---- warp-per-row path (hidden <= 2048) --------------------------------------------------------------------
constexpr int kWarpMaxH = 2048;
#define DISPATCH_NV(H, ...)                                        \
  {                                                                \
    const int need_ = ((H) / 8 + 31) / 32;                         \
    if (need_ <= 1) { constexpr int NV = 1; __VA_ARGS__ }          \
    else if (need_ <= 2) { constexpr int NV = 2; __VA_ARGS__ }     \
    else if (need_ <= 4) { constexpr int NV = 4; __VA_ARGS__ }     \
    else if (need_ <= 7) { constexpr int NV = 7; __VA_ARGS__ }     \
    else { constexpr int NV = 8; __VA_ARGS__ }                     \
  }
#define DISPATCH_16_NV(x, ...)                                     \
  if ((x).scalar_type() == torch::kBFloat16) {                     \
    using T = __nv_bfloat16;                                       \
    DISPATCH_NV((x).size(1), __VA_ARGS__)                          \
  } else {                                                         \
    using T = __half;                                              \
    DISPATCH_NV((x).size(1), __VA_ARGS__)                          \
  }

#define DISPATCH_16_NV_BWD(x, ...)                                 \
  {                                                                \
    const int need_ = ((x).size(1) / 8 + 31) / 32;                 \
    if ((x).scalar_type() == torch::kBFloat16) {                   \
      using T = __nv_bfloat16;                                     \
      DISPATCH_NV_BWD(__VA_ARGS__)                                 \
    } else {                                                       \
      using T = __half;                                            \
      DISPATCH_NV_BWD(__VA_ARGS__)                                 \
    }                                                              \
  }
#define DISPATCH_NV_BWD(...)                                       \
  if (need_ <= 1) { constexpr int NV = 1; __VA_ARGS__ }            \
  else if (need_ <= 2) { constexpr int NV = 2; __VA_ARGS__ }       \
  else if (need_ <= 4) { constexpr int NV = 4; __VA_ARGS__ }       \
  else { constexpr int NV = 5; __VA_ARGS__ }

static bool warp_path(const torch::Tensor& x) { return x.size(1) <= kWarpMaxH; }

// y = LN(x (+ residual)); returns {y, mean, rstd, sum}: `sum` is x + residual (undefined without a residual).
std::vector<torch::Tensor> layer_norm_fwd_res(torch::Tensor x, c10::optional<torch::Tensor> residual, torch::Tensor gamma,
                                              torch::Tensor beta, double eps) {
  check_rows(x);
  const bool has_res = residual.has_value() && residual->defined();
  const int rows = x.size(0), H = x.size(1);
  TORCH_CHECK((gamma.scalar_type() == torch::kFloat32 || gamma.scalar_type() == x.scalar_type()) &&
              beta.scalar_type() == gamma.scalar_type() && gamma.is_contiguous() && beta.is_contiguous() &&
              gamma.numel() == H && beta.numel() == H, "norm parameters must be contiguous [H], fp32 or of the rows' type");
  // A CTA per row for wide rows (with a residual from 1536 columns on: 32768 x 1600 104 us by warps, 96 by CTAs, 4096 x 2048 28
  // and 21; without one the warps stay ahead at 1600, 52 and 76), and for so few that eight rows per CTA leave most SMs without one (decoding: 8 rows of 2048
  // took 9.2 us on one SM, every vector of a row in the same 32 lanes; 2.4 us now).
  const bool cta = !warp_path(x) || (has_res && H > 1536) || rows <= 2 * at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  torch::Tensor sum;
  if (has_res) {
    check_rows(*residual);
    TORCH_CHECK(residual->sizes() == x.sizes() && residual->scalar_type() == x.scalar_type());
    if (cta) return layer_norm_fwd_cta(x, &*residual, gamma, beta, eps);
    sum = torch::empty_like(x);
  } else if (cta) {
    return layer_norm_fwd_cta(x, nullptr, gamma, beta, eps);
  }
  gamma = aligned16(gamma);
  beta = aligned16(beta);
  auto y = torch::empty_like(x);
  auto mean = torch::empty({rows}, x.options().dtype(torch::kFloat32));
  auto rstd = torch::empty({rows}, x.options().dtype(torch::kFloat32));
  if (rows == 0) return {y, mean, rstd, sum};
  auto stream = at::cuda::getCurrentCUDAStream();
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  const int grid = std::max(1, std::min((rows + kWarpRows - 1) / kWarpRows, sms * 6));
#define LAUNCH_LN_FWD(RES, P)                                                                                             \
  ln_fwd_warp_kernel<T, NV, RES, P><<<grid, 32 * kWarpRows, 0, stream>>>(                                                 \
      reinterpret_cast<const T*>(x.data_ptr()), RES ? reinterpret_cast<const T*>(residual->data_ptr()) : nullptr,         \
      reinterpret_cast<const P*>(gamma.data_ptr()), reinterpret_cast<const P*>(beta.data_ptr()),                          \
      RES ? reinterpret_cast<T*>(sum.data_ptr()) : nullptr, reinterpret_cast<T*>(y.data_ptr()), mean.data_ptr<float>(),   \
      rstd.data_ptr<float>(), rows, H, static_cast<float>(eps))
  const bool f32 = gamma.scalar_type() == torch::kFloat32;
  DISPATCH_16_NV(x, {
    if (has_res) { if (f32) LAUNCH_LN_FWD(true, float); else LAUNCH_LN_FWD(true, T); }
    else { if (f32) LAUNCH_LN_FWD(false, float); else LAUNCH_LN_FWD(false, T); }
  })
#undef LAUNCH_LN_FWD
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  return {y, mean, rstd, sum};
}

// {dx, dgamma, dbeta} with dx = LN'(dy) (+ dres, the gradient that reaches the normalised tensor directly).
std::vector<torch::Tensor> layer_norm_bwd_res(torch::Tensor dy, torch::Tensor x, torch::Tensor mean, torch::Tensor rstd,
                                              torch::Tensor gamma, c10::optional<torch::Tensor> dres) {
  check_rows(x);
  check_rows(dy);
  const bool has_res = dres.has_value() && dres->defined();
  if (has_res) {
    check_rows(*dres);
    TORCH_CHECK(dres->sizes() == x.sizes() && dres->scalar_type() == x.scalar_type());
  }
  const int rows = x.size(0), H = x.size(1);
  TORCH_CHECK(gamma.scalar_type() == torch::kFloat32 && gamma.is_contiguous() && gamma.numel() == H,
              "norm parameters must be contiguous fp32 [H]");
  if (H > kWarpMaxBwd) return layer_norm_bwd_cta(dy, x, mean, rstd, gamma, has_res ? &*dres : nullptr);
  gamma = aligned16(gamma);
  auto dx = torch::empty_like(x);
  auto f32 = x.options().dtype(torch::kFloat32);
  if (rows == 0) return {dx, torch::zeros({H}, f32), torch::zeros({H}, f32)};
  auto dgamma = torch::empty({H}, f32), dbeta = torch::empty({H}, f32);
  auto stream = at::cuda::getCurrentCUDAStream();
  const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
  const int grid = std::max(1, std::min((rows + kWarpRows - 1) / kWarpRows, 2 * sms));
  auto scratch = torch::empty({2, grid, H}, f32);
  float* pdg = scratch.data_ptr<float>();
  float* pdb = pdg + static_cast<size_t>(grid) * H;
  const size_t smem = static_cast<size_t>(kWarpRows) * 2 * H * sizeof(float);
  if (has_res) {
    DISPATCH_16_NV_BWD(x, (launch_ln_bwd_warp<T, NV, true>(grid, smem, stream, dy.data_ptr(), x.data_ptr(), mean.data_ptr<float>(),
                                                       rstd.data_ptr<float>(), gamma.data_ptr<float>(), dres->data_ptr(),
                                                       dx.data_ptr(), pdg, pdb, rows, H));)
  } else {
    DISPATCH_16_NV_BWD(x, (launch_ln_bwd_warp<T, NV, false>(grid, smem, stream, dy.data_ptr(), x.data_ptr(), mean.data_ptr<float>(),
                                                        rstd.data_ptr<float>(), gamma.data_ptr<float>(), nullptr, dx.data_ptr(),
                                                        pdg, pdb, rows, H));)
  }
  C10_CUDA_KERNEL_LAUNCH_CHECK();
  colsum_launch(pdg, pdb, dgamma.data_ptr<float>(), dbeta.data_ptr<float>(), grid, H, stream);
  return {dx, dgamma, dbeta};
}

}  // namespace cw
