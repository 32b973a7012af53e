// Memory-bound companions of the convolution kernels for NHWC bf16 feature maps (C a multiple of 8, 16-byte
// accesses): batch normalisation (training) fused with the residual add and ReLU, 3x3/s2 max pooling, global
// average pooling, 2x spatial subsampling and its adjoint (a 1x1 convolution with stride 2 is subsample + 1x1), and the im2col of the 7x7/s2 stem whose 3 input channels do not fill a TMA box.
//
// Reference: oneflow/user/kernels/normalization_kernel.cu (cuDNN BN + fused add/relu), pool_gpu_kernel / max_pool
// kernels, adaptive_avg_pool_gpu_kernel.cu.
#include <type_traits>

#include "../common/host_utils.h"
#include "../common/ptx.cuh"
#include "ofb_kernels.h"

namespace ofb {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void un8(const uint4& q, float (&v)[8]) {
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(w[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
  }
}
__device__ __forceinline__ void ld8(const bf16* p, float (&v)[8]) { un8(*reinterpret_cast<const uint4*>(p), v); }
__device__ __forceinline__ void st8(bf16* p, const float (&v)[8]) {
  uint4 o;
  o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
  o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
  *reinterpret_cast<uint4*>(p) = o;
}

// ------------------------------------------------------------------------------------------------ batch norm
// Two per-channel sums over all rows in one pass. MODE 0: (x, x^2). MODE 1: (g, g * xhat) with
// g = dy (* [y > 0] when relu: from the forward's mask, else from y) and xhat = (x - mean) * rstd; g_out receives g when a
// residual branch wants it as its gradient. Threads are laid out as [row lane][8-channel vector], several rows in flight each;
// a block reduces its row lanes in shared memory and adds the result to out[0..C) and out[C..2C).
template <int MODE>
__global__ void __launch_bounds__(256)
bn_reduce_kernel(const bf16* __restrict__ a, const bf16* __restrict__ x, const bf16* __restrict__ y,
                 const unsigned char* __restrict__ mask, const float* __restrict__ mean, const float* __restrict__ rstd, long long rows,
                 int C, int relu, bf16* __restrict__ g_out, float* out) {
  const int vpr = C >> 3;                       // 8-channel vectors per row
  const int vec = threadIdx.x % vpr;
  const int rlane = threadIdx.x / vpr;
  const int rlanes = blockDim.x / vpr;
  float s1[8], s2[8], mu[8], rs[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s1[j] = s2[j] = 0.f;
  if (MODE == 1) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      mu[j] = mean[vec * 8 + j];
      rs[j] = rstd[vec * 8 + j];
    }
  }
  if (rlane < rlanes) {
    // U rows: all loads first (no branch in between: with a bounds check per row the loads were not overlapped)
    auto rows_at = [&](long long r0, long long step, auto n) {
      constexpr int U = decltype(n)::value;
      uint4 qa[U];
      [[maybe_unused]] uint4 qx[MODE == 1 ? U : 1], qy[MODE == 1 ? U : 1];
      [[maybe_unused]] unsigned int bits[MODE == 1 ? U : 1];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const long long r = r0 + u * step;
        qa[u] = *reinterpret_cast<const uint4*>(a + r * C + vec * 8);
        if constexpr (MODE == 1) {
          qx[u] = *reinterpret_cast<const uint4*>(x + r * C + vec * 8);
          if (mask) bits[u] = mask[r * vpr + vec];
          else if (relu) qy[u] = *reinterpret_cast<const uint4*>(y + r * C + vec * 8);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float v[8];
        un8(qa[u], v);
        if constexpr (MODE == 0) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            s1[j] += v[j];
            s2[j] += v[j] * v[j];
          }
        } else {
          float xv[8];
          un8(qx[u], xv);
          if (mask) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = (bits[u] >> j) & 1u ? v[j] : 0.f;
          } else if (relu) {
            float yv[8];
            un8(qy[u], yv);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = yv[j] > 0.f ? v[j] : 0.f;
          }
          if (g_out) st8(g_out + (r0 + u * step) * C + vec * 8, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            s1[j] += v[j];
            s2[j] += v[j] * (xv[j] - mu[j]) * rs[j];
          }
        }
      }
    };
    constexpr int U = MODE == 0 ? 1 : 4;      // one stream: the compiler overlaps the rounds by itself (four rows by hand: 108 against 67 us)
    const long long step = (long long)gridDim.x * rlanes;
    long long r0 = blockIdx.x * (long long)rlanes + rlane;
    for (; r0 + (U - 1) * step < rows; r0 += U * step) rows_at(r0, step, std::integral_constant<int, U>());
    for (; r0 < rows; r0 += step) rows_at(r0, step, std::integral_constant<int, 1>());
  }
  __shared__ float red[256 * 16];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    red[threadIdx.x * 16 + j] = s1[j];
    red[threadIdx.x * 16 + 8 + j] = s2[j];
  }
  __syncthreads();
  // thread t < vpr * 16 sums one (vector, component) over the row lanes
  for (int i = threadIdx.x; i < vpr * 16; i += blockDim.x) {
    const int v = i / 16, comp = i % 16;
    float t = 0.f;
    for (int l = 0; l < rlanes; ++l) t += red[(l * vpr + v) * 16 + comp];
    atomicAdd(&out[(comp >> 3) * C + v * 8 + (comp & 7)], t);
  }
}

// sums[0..C) = sum x, sums[C..2C) = sum x^2  ->  mean, rstd, the folded affine map y = scale * x + shift
// (scale = gamma * rstd, shift = beta - mean * scale), and the running statistics when given.
__global__ void bn_finalize_kernel(const float* __restrict__ sums, float inv_rows, float eps, float momentum, float unbias, int C,
                                   const float* __restrict__ gamma, const float* __restrict__ beta, float* mean, float* rstd, float* scale,
                                   float* shift, float* running_mean, float* running_var) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const float m = sums[c] * inv_rows;
  const float var = fmaxf(sums[C + c] * inv_rows - m * m, 0.f);
  const float rs = rsqrtf(var + eps);
  mean[c] = m;
  rstd[c] = rs;
  const float sc = gamma[c] * rs;
  scale[c] = sc;
  shift[c] = beta[c] - m * sc;
  if (running_mean) {
    running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * m;
    running_var[c] = (1.f - momentum) * running_var[c] + momentum * var * unbias;
  }
}

// Backward coefficients per channel: dx = a * g + b * x + c with
//   a = gamma rstd,  b = -a rstd s2 / rows,  c = -a s1 / rows - b mean      (s1 = sum g, s2 = sum g xhat)
// and the parameter gradients dgamma = s2, dbeta = s1 where wanted (added to what is there with acc_*). A kernel of its own: the
// element pass with this work at the start of its blocks was slower by more than the launch (802816 x 64: 65 instead of 49 + 2 us).
__global__ void bn_bwd_coeffs_kernel(const float* __restrict__ sums, const float* __restrict__ mean, const float* __restrict__ rstd,
                                     const float* __restrict__ gamma, float inv_rows, int C, float* coef, float* dgamma, int acc_gamma,
                                     float* dbeta, int acc_beta) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const float a = gamma[c] * rstd[c];
  const float b = -a * rstd[c] * sums[C + c] * inv_rows;
  coef[c] = a;
  coef[C + c] = b;
  coef[2 * C + c] = -a * sums[c] * inv_rows - b * mean[c];
  if (dgamma) dgamma[c] = acc_gamma ? dgamma[c] + sums[C + c] : sums[C + c];
  if (dbeta) dbeta[c] = acc_beta ? dbeta[c] + sums[c] : sums[c];
}

// Streaming kernels below: when the 8-channel vectors per row divide the block size, a thread keeps the same
// channels for every row it visits, so the per-channel coefficients are loaded into registers once.
__device__ __forceinline__ void load_coef8(const float* p, float (&v)[8]) {
  const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
  v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
  v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
}

// y = [relu](scale * x + shift [+ residual]). `mask` receives one byte per eight channels, bit j = (y of channel j > 0): what the
// backward needs of y, at a sixteenth of its bytes.
__global__ void __launch_bounds__(256)
bn_apply_kernel(const bf16* __restrict__ x, const bf16* __restrict__ residual, const float* __restrict__ scale,
                const float* __restrict__ shift, long long vecs, int C, int relu, bf16* __restrict__ y, unsigned char* __restrict__ mask) {
  const int vpr = C >> 3;
  const bool fixed = (blockDim.x % vpr) == 0;
  float sc[8], sh[8];
  if (fixed) {
    load_coef8(scale + (threadIdx.x % vpr) * 8, sc);
    load_coef8(shift + (threadIdx.x % vpr) * 8, sh);
  }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < vecs; i += (long long)gridDim.x * blockDim.x) {
    if (!fixed) {
      const int c0 = static_cast<int>(i % vpr) * 8;
      load_coef8(scale + c0, sc);
      load_coef8(shift + c0, sh);
    }
    float v[8];
    ld8(x + i * 8, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = fmaf(v[j], sc[j], sh[j]);
    if (residual) {
      float r[8];
      ld8(residual + i * 8, r);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += r[j];
    }
    if (relu) {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = fmaxf(v[j], 0.f);
    }
    if (mask) {
      unsigned int bits = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) bits |= (__bfloat162float(__float2bfloat16(v[j])) > 0.f ? 1u : 0u) << j;
      mask[i] = static_cast<unsigned char>(bits);
    }
    st8(y + i * 8, v);
  }
}

// dx = a * g + b * x + c, g = dy (* [y > 0], from y or from the forward's mask). coef = [a | b | c], each C long. (A residual
// branch takes g as its gradient: then the reduction has written it and this pass reads it as dy, without y.)
__global__ void __launch_bounds__(256)
bn_bwd_apply_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ y,
                    const unsigned char* __restrict__ mask, const float* __restrict__ coef, long long vecs, int C, int relu,
                    bf16* __restrict__ dx) {
  const int vpr = C >> 3;
  const bool fixed = (blockDim.x % vpr) == 0;
  float ca[8], cb[8], cc[8];
  if (fixed) {
    const int c0 = (threadIdx.x % vpr) * 8;
    load_coef8(coef + c0, ca);
    load_coef8(coef + C + c0, cb);
    load_coef8(coef + 2 * C + c0, cc);
  }
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < vecs; i += (long long)gridDim.x * blockDim.x) {
    if (!fixed) {
      const int c0 = static_cast<int>(i % vpr) * 8;
      load_coef8(coef + c0, ca);
      load_coef8(coef + C + c0, cb);
      load_coef8(coef + 2 * C + c0, cc);
    }
    float g[8], xv[8];
    ld8(dy + i * 8, g);
    ld8(x + i * 8, xv);
    if (relu && mask) {
      const unsigned int bits = mask[i];
#pragma unroll
      for (int j = 0; j < 8; ++j) g[j] = (bits >> j) & 1u ? g[j] : 0.f;
    } else if (relu) {
      float yv[8];
      ld8(y + i * 8, yv);
#pragma unroll
      for (int j = 0; j < 8; ++j) g[j] = yv[j] > 0.f ? g[j] : 0.f;
    }
    float o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = fmaf(ca[j], g[j], fmaf(cb[j], xv[j], cc[j]));
    st8(dx + i * 8, o);
  }
}

// ------------------------------------------------------------------------------------------------ pooling
// 3x3 window, stride 2, padding 1. idx keeps the winning tap (0..8) for the backward.
template <typename I>
__global__ void __launch_bounds__(256)
maxpool_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, unsigned char* __restrict__ idx, int N, int H, int W, int C, int OH,
                   int OW) {
  const int vpr = C >> 3;
  const I total = static_cast<I>(N) * OH * OW * vpr;
  for (I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; i < total; i += static_cast<I>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % static_cast<I>(vpr));
    I p = i / static_cast<I>(vpr);
    const int ow = static_cast<int>(p % static_cast<I>(OW));
    p /= static_cast<I>(OW);
    const int oh = static_cast<int>(p % static_cast<I>(OH));
    const int n = static_cast<int>(p / OH);
    float best[8];
    unsigned char bi[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      best[j] = -3.0e38f;
      bi[j] = 4;
    }
    for (int r = 0; r < 3; ++r) {
      const int h = 2 * oh + r - 1;
      if (h < 0 || h >= H) continue;
      for (int s = 0; s < 3; ++s) {
        const int w = 2 * ow + s - 1;
        if (w < 0 || w >= W) continue;
        float t[8];
        ld8(x + ((static_cast<long long>(n) * H + h) * W + w) * C + v * 8, t);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (t[j] > best[j]) {
            best[j] = t[j];
            bi[j] = static_cast<unsigned char>(r * 3 + s);
          }
      }
    }
    st8(y + static_cast<long long>(i) * 8, best);
    uint2 packed;
    packed.x = bi[0] | (bi[1] << 8) | (bi[2] << 16) | (bi[3] << 24);
    packed.y = bi[4] | (bi[5] << 8) | (bi[6] << 16) | (bi[7] << 24);
    *reinterpret_cast<uint2*>(idx + static_cast<long long>(i) * 8) = packed;
  }
}

// Gather form of the backward. A thread owns a 2 x 2 block of input pixels (rows 2a, 2a + 1, columns 2b, 2b + 1), which the four
// windows (a..a+1, b..b+1) cover: each window is read once for the block (a thread per pixel read nine windows for the same four).
// 256 x 112 x 112 x 64: 374 -> 143 us (a copy of the same bytes takes 86).
template <typename I>
__global__ void __launch_bounds__(256)
maxpool_bwd_kernel(const bf16* __restrict__ dy, const unsigned char* __restrict__ idx, bf16* __restrict__ dx, int N, int H, int W, int C,
                   int OH, int OW) {
  const int vpr = C >> 3;
  const I total = static_cast<I>(N) * OH * OW * vpr;      // OH = ceil(H / 2), OW = ceil(W / 2): one block per window corner
  for (I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; i < total; i += static_cast<I>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % static_cast<I>(vpr));
    I p = i / static_cast<I>(vpr);
    const int b = static_cast<int>(p % static_cast<I>(OW));
    p /= static_cast<I>(OW);
    const int a = static_cast<int>(p % static_cast<I>(OH));
    const long long n = p / static_cast<I>(OH);
    uint2 tap[2][2];
    uint4 g[2][2];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        tap[u][w] = make_uint2(0xFFFFFFFFu, 0xFFFFFFFFu);      // a window outside matches no tap
        g[u][w] = make_uint4(0, 0, 0, 0);
        if (a + u < OH && b + w < OW) {
          const long long o = ((n * OH + a + u) * OW + b + w) * vpr + v;
          tap[u][w] = *reinterpret_cast<const uint2*>(idx + o * 8);
          g[u][w] = *reinterpret_cast<const uint4*>(dy + o * 8);
        }
      }
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        if (2 * a + u >= H || 2 * b + w >= W) continue;
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
        // pixel (2a + u, 2b + w) is tap (1 + u - 2 du, 1 + w - 2 dw) of window (a + du, b + dw), du <= u, dw <= w
#pragma unroll
        for (int du = 0; du <= u; ++du)
#pragma unroll
          for (int dw = 0; dw <= w; ++dw) {
            const unsigned int want = (1 + u - 2 * du) * 3 + (1 + w - 2 * dw);
            float gv[8];
            un8(g[du][dw], gv);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const unsigned int t = ((j < 4 ? tap[du][dw].x : tap[du][dw].y) >> (8 * (j & 3))) & 0xffu;
              if (t == want) acc[j] += gv[j];
            }
          }
        st8(dx + (((n * H + 2 * a + u) * W + 2 * b + w) * vpr + v) * 8, acc);
      }
  }
}

// mean over the HW pixels of each image: x [N, HW, C] -> y [N, C]; backward broadcasts dy / HW.
__global__ void __launch_bounds__(256)
avgpool_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, int N, int HW, int C) {
  const int vpr = C >> 3;
  const long long total = static_cast<long long>(N) * vpr;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int v = static_cast<int>(i % vpr);
    const long long n = i / vpr;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int p = 0; p < HW; ++p) {
      float t[8];
      ld8(x + (n * HW + p) * C + v * 8, t);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += t[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] *= 1.f / HW;
    st8(y + i * 8, acc);
  }
}
template <typename I>
__global__ void __launch_bounds__(256)
avgpool_bwd_kernel(const bf16* __restrict__ dy, bf16* __restrict__ dx, int N, int HW, int C) {
  const int vpr = C >> 3;
  const I total = static_cast<I>(N) * HW * vpr;
  for (I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; i < total; i += static_cast<I>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % static_cast<I>(vpr));
    const long long n = i / static_cast<I>(vpr) / HW;
    float g[8];
    ld8(dy + (n * vpr + v) * 8, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] *= 1.f / HW;
    st8(dx + static_cast<long long>(i) * 8, g);
  }
}

// ------------------------------------------------------------------------------------------------ stride 2 helpers
// y[n, oh, ow] = x[n, 2 oh, 2 ow]  (adjoint: dx = 0 except dx[n, 2 oh, 2 ow] = dy[n, oh, ow])
template <typename I>
__global__ void __launch_bounds__(256)
subsample2_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, int N, int H, int W, int C, int OH, int OW) {
  const int vpr = C >> 3;
  const I total = static_cast<I>(N) * OH * OW * vpr;
  for (I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; i < total; i += static_cast<I>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % static_cast<I>(vpr));
    I p = i / static_cast<I>(vpr);
    const int ow = static_cast<int>(p % static_cast<I>(OW));
    p /= static_cast<I>(OW);
    const int oh = static_cast<int>(p % static_cast<I>(OH));
    const long long n = p / static_cast<I>(OH);
    reinterpret_cast<uint4*>(y)[i] = *reinterpret_cast<const uint4*>(x + ((n * H + 2 * oh) * W + 2 * ow) * C + v * 8);
  }
}
template <typename I>
__global__ void __launch_bounds__(256)
upsample2_zero_kernel(const bf16* __restrict__ dy, bf16* __restrict__ dx, int N, int H, int W, int C, int OH, int OW) {
  const int vpr = C >> 3;
  const I total = static_cast<I>(N) * H * W * vpr;
  for (I i = blockIdx.x * static_cast<I>(blockDim.x) + threadIdx.x; i < total; i += static_cast<I>(gridDim.x) * blockDim.x) {
    const int v = static_cast<int>(i % static_cast<I>(vpr));
    I p = i / static_cast<I>(vpr);
    const int w = static_cast<int>(p % static_cast<I>(W));
    p /= static_cast<I>(W);
    const int h = static_cast<int>(p % static_cast<I>(H));
    const long long n = p / static_cast<I>(H);
    uint4 q = make_uint4(0, 0, 0, 0);
    if (!(h & 1) && !(w & 1) && (h >> 1) < OH && (w >> 1) < OW)
      q = *reinterpret_cast<const uint4*>(dy + ((n * OH + (h >> 1)) * OW + (w >> 1)) * C + v * 8);
    reinterpret_cast<uint4*>(dx)[i] = q;
  }
}

// cols[(n, oh, ow)][(r * S + s) * Cin + c] = x[n, stride oh + r - pad, stride ow + s - pad, c] (zero outside and in
// the padding columns up to ldc). For small Cin (the RGB stem). A CTA takes `cpp` neighbouring output columns of one output row
// (n, oh): the R pieces of input rows that they see lie zero-padded in shared memory, where the S Cin values of one filter row are
// neighbours, and every thread gathers 8 columns of the matrix at a time. (A thread that fetched its 8 values from global memory
// after 64-bit divisions: 996 us for 256 x 224 x 224 x 3, 7 x 7, against 463 us; 976 MB are written, 149 us at the copy rate.)
// CIN_ / R_ / S_ > 0 fix the shape at compile time (constant divisors); 0 takes the runtime values. STAGED = false reads the image
// directly: windows too large for shared memory, and small problems.
template <int CIN_, int R_, int S_, bool STAGED>
__global__ void __launch_bounds__(256)
im2col_small_kernel(const bf16* __restrict__ x, bf16* __restrict__ cols, int H, int W, int Cin_rt, int R_rt, int S_rt, int stride, int pad,
                    int OH, int OW, int cpp, int ldc) {
  extern __shared__ unsigned short rows_s[];            // [R][(stride (cpp - 1) + S) Cin]
  const int Cin = CIN_ > 0 ? CIN_ : Cin_rt, R = R_ > 0 ? R_ : R_rt, S = S_ > 0 ? S_ : S_rt;
  const int ow0 = blockIdx.y * cpp, n_ow = min(cpp, OW - ow0);
  const int oh = blockIdx.x % OH;
  const long long n = blockIdx.x / OH;
  const int from = stride * ow0 * Cin, rlen = (stride * (n_ow - 1) + S) * Cin, lo = pad * Cin, hi = lo + W * Cin;
  // element i of the piece of zero-padded input row r
  auto fetch = [&](int r, int i) -> unsigned short {
    const int h = stride * oh + r - pad;
    const bool in = h >= 0 && h < H && from + i >= lo && from + i < hi;
    return in ? reinterpret_cast<const unsigned short*>(x)[(n * H + h) * W * Cin + (from + i - lo)] : static_cast<unsigned short>(0);
  };
  if constexpr (STAGED) {
    for (int r = 0; r < R; ++r)
      for (int i = threadIdx.x; i < rlen; i += blockDim.x) rows_s[r * rlen + i] = fetch(r, i);
    __syncthreads();
  }
  const int vpr = ldc >> 3, fr = S * Cin, kcols = R * fr;
  uint4* out = reinterpret_cast<uint4*>(cols) + (static_cast<long long>(blockIdx.x) * OW + ow0) * vpr;
  for (int i = threadIdx.x; i < n_ow * vpr; i += blockDim.x) {
    const int ow = i / vpr, col0 = (i - ow * vpr) * 8;
    const int first = stride * ow * Cin;
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int col = col0 + j, r = col / fr;
      uint32_t val = 0;
      if (col < kcols) val = STAGED ? rows_s[r * rlen + first + (col - r * fr)] : fetch(r, first + (col - r * fr));
      if (j & 1) o[j >> 1] |= val << 16;
      else o[j >> 1] = val;
    }
    out[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace ofb

using namespace ofb;

static inline int aux_grid(long long items) {
  long long b = (items + 255) / 256;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return static_cast<int>(b);
}

// The index kernels split a vector's number into its coordinates; below 2^31 vectors with 32-bit divisions
// (a pooling backward with a thread per pixel, 256 x 112 x 112 x 64: 374 us, with 64-bit divisions 418 us).
#define OFB_AUX_LAUNCH(kern, items, ...)                                                             \
  do {                                                                                               \
    const long long items_ = (items);                                                                \
    if (items_ < (1ll << 31)) kern<unsigned int><<<aux_grid(items_), 256, 0, (cudaStream_t)stream>>>(__VA_ARGS__); \
    else kern<long long><<<aux_grid(items_), 256, 0, (cudaStream_t)stream>>>(__VA_ARGS__);           \
  } while (0)

// sums [2 C] fp32 must be zero on entry. mode 0: sums of x and x^2 (pass x as `a`). mode 1: sums of g and g * xhat; with relu the
// sign of the forward's output comes from `mask` (ofb_bn_apply) or, when that is null, from y; g_out (may be null) receives g.
OFB_API int ofb_bn_reduce(int mode, const void* a, const void* x, const void* y, const void* mask, const float* mean, const float* rstd,
                          long long rows, int C, int relu, void* g_out, float* sums, void* stream) {
  if (C % 8 || C > 2048) return fail("bn: channels must be a multiple of 8, at most 2048");
  if (rows == 0) return 0;
  const int vpr = C / 8;
  const int rlanes = 256 / vpr;
  long long blocks = (rows + rlanes * 16 - 1) / (rlanes * 16);
  // few blocks: every one of them ends in 2 C atomic additions (12544 x 2048, mode 0: 27 us with eight blocks per SM, 20 with three)
  const int per_sm = mode == 0 ? 3 : 2;
  if (blocks > 148 * per_sm) blocks = 148 * per_sm;
  if (blocks < 1) blocks = 1;
  if (mode == 0)
    bn_reduce_kernel<0><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)a, nullptr, nullptr, nullptr, nullptr, nullptr, rows,
                                                                         C, 0, nullptr, sums);
  else
    bn_reduce_kernel<1><<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)a, (const bf16*)x, (const bf16*)y,
                                                                         relu ? (const unsigned char*)mask : nullptr, mean, rstd, rows, C, relu, (bf16*)g_out,
                                                                         sums);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

OFB_API int ofb_bn_finalize(const float* sums, long long rows, float eps, float momentum, int C, const float* gamma, const float* beta,
                            float* mean, float* rstd, float* scale, float* shift, float* running_mean, float* running_var, void* stream) {
  const float unbias = rows > 1 ? static_cast<float>(rows) / static_cast<float>(rows - 1) : 1.f;
  bn_finalize_kernel<<<(C + 127) / 128, 128, 0, (cudaStream_t)stream>>>(sums, 1.f / rows, eps, momentum, unbias, C, gamma, beta, mean, rstd,
                                                                       scale, shift, running_mean, running_var);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

// y = [relu](scale * x + shift [+ residual]) with per-channel fp32 scale / shift; mask [rows * C / 8] bytes or null.
OFB_API int ofb_bn_apply(const void* x, const void* residual, const float* scale, const float* shift, long long rows, int C, int relu,
                         void* y, void* mask, void* stream) {
  if (C % 8) return fail("bn: channels must be a multiple of 8");
  const long long vecs = rows * (C / 8);
  if (vecs == 0) return 0;
  bn_apply_kernel<<<aux_grid(vecs), 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (const bf16*)residual, scale, shift, vecs, C, relu,
                                                                  (bf16*)y, (unsigned char*)mask);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

// coef [3 C] is scratch written here. sums = [sum g | sum g xhat] from ofb_bn_reduce(mode 1). dgamma / dbeta [C] (may be null) receive
// the parameter gradients, added to what is there with acc_gamma / acc_beta.
OFB_API int ofb_bn_bwd_apply(const void* dy, const void* x, const void* y, const void* mask, const float* mean, const float* rstd,
                             const float* gamma, const float* sums, float* coef, long long rows, int C, int relu, float* dgamma, int acc_gamma,
                             float* dbeta, int acc_beta, void* dx, void* stream) {
  if (C % 8) return fail("bn: channels must be a multiple of 8");
  const long long vecs = rows * (C / 8);
  if (C == 0 || (vecs == 0 && !dgamma && !dbeta)) return 0;
  bn_bwd_coeffs_kernel<<<(C + 127) / 128, 128, 0, (cudaStream_t)stream>>>(sums, mean, rstd, gamma, 1.f / rows, C, coef, dgamma, acc_gamma, dbeta,
                                                                        acc_beta);
  OFB_CUDA_OK(cudaGetLastError());
  if (vecs == 0) return 0;
  bn_bwd_apply_kernel<<<aux_grid(vecs), 256, 0, (cudaStream_t)stream>>>((const bf16*)dy, (const bf16*)x, (const bf16*)y,
                                                                      (const unsigned char*)mask, coef, vecs, C, relu, (bf16*)dx);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}

OFB_API int ofb_maxpool3x3s2_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C, void* stream) {
  if (C % 8) return fail("maxpool: channels must be a multiple of 8");
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  OFB_AUX_LAUNCH(maxpool_fwd_kernel, (long long)N * OH * OW * (C / 8), (const bf16*)x, (bf16*)y, (unsigned char*)idx, N, H, W, C, OH, OW);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
OFB_API int ofb_maxpool3x3s2_bwd(const void* dy, const void* idx, void* dx, int N, int H, int W, int C, void* stream) {
  if (C % 8) return fail("maxpool: channels must be a multiple of 8");
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  OFB_AUX_LAUNCH(maxpool_bwd_kernel, (long long)N * OH * OW * (C / 8), (const bf16*)dy, (const unsigned char*)idx, (bf16*)dx, N, H, W, C, OH, OW);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
OFB_API int ofb_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream) {
  if (C % 8) return fail("avgpool: channels must be a multiple of 8");
  avgpool_fwd_kernel<<<aux_grid((long long)N * (C / 8)), 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)y, N, HW, C);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
OFB_API int ofb_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream) {
  if (C % 8) return fail("avgpool: channels must be a multiple of 8");
  OFB_AUX_LAUNCH(avgpool_bwd_kernel, (long long)N * HW * (C / 8), (const bf16*)dy, (bf16*)dx, N, HW, C);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
OFB_API int ofb_subsample2(const void* x, void* y, int N, int H, int W, int C, void* stream) {
  if (C % 8) return fail("subsample: channels must be a multiple of 8");
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  OFB_AUX_LAUNCH(subsample2_kernel, (long long)N * OH * OW * (C / 8), (const bf16*)x, (bf16*)y, N, H, W, C, OH, OW);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
OFB_API int ofb_upsample2_zero(const void* dy, void* dx, int N, int H, int W, int C, void* stream) {
  if (C % 8) return fail("upsample: channels must be a multiple of 8");
  const int OH = (H + 1) / 2, OW = (W + 1) / 2;
  OFB_AUX_LAUNCH(upsample2_zero_kernel, (long long)N * H * W * (C / 8), (const bf16*)dy, (bf16*)dx, N, H, W, C, OH, OW);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
OFB_API int ofb_im2col_small(const void* x, void* cols, int N, int H, int W, int Cin, int R, int S, int stride, int pad, int ldc,
                             void* stream) {
  if (ldc % 8 || ldc < R * S * Cin) return fail("im2col: leading dimension must be a multiple of 8 covering R S Cin");
  const int OH = (H + 2 * pad - R) / stride + 1, OW = (W + 2 * pad - S) / stride + 1;
  if (N <= 0 || OH <= 0 || OW <= 0 || ldc == 0) return 0;
  const long long rows = (long long)N * OH;
  if (rows > 0x7FFFFFFFll) return fail("im2col: too many output rows");
  // Output columns of a CTA: one round of its threads for small problems, which read the image through L1 and do without the wait
  // between staging and gathering (1 x 96 x 96 2.7 against 3.7 us, 4 x 224 x 224 12.8 against 14.1; 32 x 96 x 96 18.2 against 16.4,
  // 256 x 224 x 224 690 against 466). Staged: whole rows from two CTAs an SM on, else pieces that make four, and never more than
  // 48 KiB of input, which every device gives without asking.
  const int round = 256 / (ldc / 8) > 0 ? 256 / (ldc / 8) : 1;
  const bool small = rows * OW * (ldc / 8) <= 1 << 20;
  int cpp = small ? round : rows < 2 * 148 ? (int)((OW * rows - 1) / (4 * 148) + 1) : OW;
  if (cpp < round || cpp > OW) cpp = round < OW ? round : OW;
  const long long fit = (48 * 1024 / (R * Cin > 0 ? 2ll * R * Cin : 1) - S) / stride + 1;      // 0 or less: not one window
  const bool staged = !small && 2ll * R * S * Cin <= 48 * 1024 && (OW - 1) / (cpp < fit ? cpp : fit) < 65535;
  if (staged && cpp > fit) cpp = (int)fit;
  if (!staged && (OW - 1) / cpp >= 65535) cpp = OW;
  auto launch = [&](auto kern, long long bytes) {
    kern<<<dim3((unsigned int)rows, (OW - 1) / cpp + 1), 256, (size_t)bytes, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)cols, H, W,
                                                                                                     Cin, R, S, stride, pad, OH, OW, cpp, ldc);
  };
  const long long smem = 2ll * R * (stride * (cpp - 1ll) + S) * Cin;
  const bool stem = Cin == 3 && R == 7 && S == 7;
  if (!staged) stem ? launch(im2col_small_kernel<3, 7, 7, false>, 0) : launch(im2col_small_kernel<0, 0, 0, false>, 0);
  else stem ? launch(im2col_small_kernel<3, 7, 7, true>, smem) : launch(im2col_small_kernel<0, 0, 0, true>, smem);
  OFB_CUDA_OK(cudaGetLastError());
  return 0;
}
