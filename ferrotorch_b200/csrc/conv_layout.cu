// Layout kernels around the shifted-row convolution GEMMs (gemm_tcgen05.cu, MODE 1 / 2) for NHWC
// bf16 activations:
//   * embed: copy [N, H, W, C] into a zeroed [N, Hp, Wp, C] grid at offset (oh, ow), optionally
//     splitting the padded image into its four stride-2 parity planes (the layout in which a
//     stride-2 filter tap is again a constant row shift);
//   * crop:  the inverse for a GEMM output -- take [N, Ho, Wo, C] out of the padded grid;
//   * im2col for filters whose channel count is not a multiple of 64 (the 3-channel stem of a
//     ResNet): rows of [KH*KW*C] patches, zero-padded to a row length that TMA can address.
// The reference writes an im2col buffer for every convolution (ferrotorch-gpu/src/conv.rs:239-520);
// here only the stem does.
#include "ft_host.h"
#include "ft_ptx.cuh"

namespace ft {

// One thread per 16-byte vector (8 channels) of the destination grid.
// planes == 1: dst[n, i, j, :] = src[n, i - oh, j - ow, :] (zero outside).
// planes == 4: dst[(a, b), n, i, j, :] = padded[n, 2 i + a, 2 j + b, :], padded as above
//              (Hp, Wp are then the plane extents, i.e. half the padded image).
__global__ void conv_embed_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int N, int H, int W,
                                  int Cv, int Hp, int Wp, int oh, int ow, int planes) {
  const long long total = static_cast<long long>(planes) * N * Hp * Wp * Cv;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % Cv);
    long long r = i / Cv;
    const int j = static_cast<int>(r % Wp); r /= Wp;
    const int ii = static_cast<int>(r % Hp); r /= Hp;
    const int n = static_cast<int>(r % N);
    const int pl = static_cast<int>(r / N);
    int hi, wi;
    if (planes == 4) {
      hi = 2 * ii + (pl >> 1) - oh;
      wi = 2 * j + (pl & 1) - ow;
    } else {
      hi = ii - oh;
      wi = j - ow;
    }
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (hi >= 0 && hi < H && wi >= 0 && wi < W)
      v = __ldg(src + ((static_cast<long long>(n) * H + hi) * W + wi) * Cv + c);
    dst[i] = v;
  }
}

// dst[n, i, j, :] = src[n, i + oh, j + ow, :] for a [N, Hp, Wp, C] source grid (bf16 or fp32,
// moved as 16-byte vectors).
__global__ void conv_crop_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int N, int Ho, int Wo,
                                 int Cv, int Hp, int Wp, int oh, int ow) {
  const long long total = static_cast<long long>(N) * Ho * Wo * Cv;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % Cv);
    long long r = i / Cv;
    const int j = static_cast<int>(r % Wo); r /= Wo;
    const int ii = static_cast<int>(r % Ho);
    const int n = static_cast<int>(r / Ho);
    dst[i] = __ldg(src + ((static_cast<long long>(n) * Hp + ii + oh) * Wp + j + ow) * Cv + c);
  }
}

// out[m, (kh * KW + kw) * C + c] = x[n, ho * s - ph + kh * d, wo * s - pw + kw * d, c]; columns
// [KH*KW*C, Kpad) are zero.  One thread per (row, tap).
__global__ void im2col_nhwc_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out, int N, int H,
                                   int W, int C, int KH, int KW, int stride, int ph, int pw, int dil, int Ho, int Wo,
                                   int Kpad) {
  const int taps = KH * KW;
  const long long total = static_cast<long long>(N) * Ho * Wo * (taps + 1);
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int tap = static_cast<int>(i % (taps + 1));
    const long long m = i / (taps + 1);
    __nv_bfloat16* row = out + m * Kpad;
    if (tap == taps) {  // the zero tail of the row
      for (int k = taps * C; k < Kpad; ++k) row[k] = __float2bfloat16(0.f);
      continue;
    }
    const int wo = static_cast<int>(m % Wo), ho = static_cast<int>((m / Wo) % Ho);
    const int n = static_cast<int>(m / (static_cast<long long>(Wo) * Ho));
    const int kh = tap / KW, kw = tap - kh * KW;
    const int hi = ho * stride - ph + kh * dil, wi = wo * stride - pw + kw * dil;
    const bool in = hi >= 0 && hi < H && wi >= 0 && wi < W;
    const __nv_bfloat16* src = x + ((static_cast<long long>(n) * H + hi) * W + wi) * C;
    if ((C & 3) == 0) {
      // 8-byte vectors: a pixel of C channels and its slot in the row are both 8-byte aligned
      const uint2* s2 = reinterpret_cast<const uint2*>(src);
      uint2* d2 = reinterpret_cast<uint2*>(row + tap * C);
      for (int c = 0; c < (C >> 2); ++c) d2[c] = in ? __ldg(s2 + c) : make_uint2(0u, 0u);
    } else {
      for (int c = 0; c < C; ++c) row[tap * C + c] = in ? src[c] : __float2bfloat16(0.f);
    }
  }
}

// Patch rows of images with four channels (an RGB image padded by one): a warp builds a row, a lane two taps, one 16-byte store.  With
// one thread per tap and 64-bit index divisions in each, 256 x 112 x 112 rows of 200 took 1.31 ms; writing them takes 0.2.
__global__ void __launch_bounds__(256)
im2col_c4_kernel(const uint2* __restrict__ x, uint4* __restrict__ out, int N, int H, int W, int KH, int KW, int stride, int ph, int pw, int dil,
                 int Ho, int Wo, int row_vecs) {
  // A warp takes sixteen pixels of an output line at a time: where a lane's two taps lie, and whether their image row exists, is found once
  // for all of them (with these divisions for every row a ResNet-50 step of 256 images took 31.72 ms, 30.95 now).
  constexpr int RUN = 16;
  const int lane = threadIdx.x & 31, taps = KH * KW, runs = (Wo + RUN - 1) / RUN;
  const int units = N * Ho * runs, step = gridDim.x * (blockDim.x >> 5);
  for (int u = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); u < units; u += step) {
    const int line = u / runs, n = line / Ho, wo0 = (u - line * runs) * RUN, count = min(RUN, Wo - wo0);
    const int h0 = (line - n * Ho) * stride - ph, w0 = wo0 * stride - pw;
    const uint2* image = x + static_cast<long long>(n) * H * W;
    for (int v = lane; v < row_vecs; v += 32) {
      const uint2* row[2];
      int w[2];
      bool there[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int tap = 2 * v + i, kh = tap / KW, h = h0 + kh * dil;
        there[i] = tap < taps && h >= 0 && h < H;
        row[i] = image + (there[i] ? h * W : 0);
        w[i] = w0 + (tap - kh * KW) * dil;
      }
      uint4* to = out + (static_cast<long long>(line) * Wo + wo0) * row_vecs + v;
#pragma unroll 4
      for (int m = 0; m < count; ++m) {
        uint2 q[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int at = w[i] + m * stride;
          q[i] = there[i] && at >= 0 && at < W ? __ldg(row[i] + at) : make_uint2(0u, 0u);
        }
        to[static_cast<long long>(m) * row_vecs] = make_uint4(q[0].x, q[0].y, q[1].x, q[1].y);
      }
    }
  }
}

// dst[i0, i1, i2] (+)= src[i0, i1, i2] between any strides and types (0 bf16, 1 fp32): filters into the rows that the GEMMs read, filter
// gradients into the parameter's layout.  order: which place of src along dimension order_dim each index of dst means.
struct FilterCopy {
  int n[3];
  long long ss[3], ds[3];
  int src_f32, dst_f32, accumulate, order_dim;
  unsigned char order[64];
};
__global__ void __launch_bounds__(256)
filter_copy_kernel(const void* __restrict__ src, void* __restrict__ dst, const FilterCopy f) {
  const int total = f.n[0] * f.n[1] * f.n[2];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int r = i / f.n[2], at[3] = {r / f.n[1], r % f.n[1], i - r * f.n[2]};
    long long s = 0, d = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s += f.ss[k] * (k == f.order_dim ? f.order[at[k]] : at[k]);
      d += f.ds[k] * at[k];
    }
    float v = f.src_f32 ? static_cast<const float*>(src)[s] : __bfloat162float(static_cast<const __nv_bfloat16*>(src)[s]);
    if (f.dst_f32) {
      float* o = static_cast<float*>(dst) + d;
      *o = f.accumulate ? *o + v : v;
    } else {
      __nv_bfloat16* o = static_cast<__nv_bfloat16*>(dst) + d;
      // what was an addition of a bf16 gradient stays one
      *o = f.accumulate ? __float2bfloat16(__bfloat162float(*o) + __bfloat162float(__float2bfloat16(v))) : __float2bfloat16(v);
    }
  }
}

static inline int layout_grid(long long work, int device) {
  const long long blocks = (work + 255) / 256;
  const long long cap = static_cast<long long>(sm_count(device)) * 16;
  return static_cast<int>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

}  // namespace ft

using namespace ft;

// src [N, H, W, C] -> dst [planes, N, Hp, Wp, C] (planes 1 or 4), see conv_embed_kernel.
// elt_bytes: 2 (bf16) or 4 (fp32); C * elt_bytes must be a multiple of 16.
FT_API int ft_conv_embed(const void* src, void* dst, int N, int H, int W, int C, int Hp, int Wp, int oh, int ow,
                         int planes, int elt_bytes, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  FT_REQUIRE(src && dst, "ft_conv_embed: null pointer");
  FT_REQUIRE(N > 0 && H > 0 && W > 0 && C > 0 && Hp > 0 && Wp > 0 && (planes == 1 || planes == 4),
             "ft_conv_embed: bad geometry");
  FT_REQUIRE((elt_bytes == 2 || elt_bytes == 4) && (C * elt_bytes) % 16 == 0,
             "ft_conv_embed: a pixel (%d channels x %d bytes) must be a multiple of 16 bytes", C, elt_bytes);
  FT_REQUIRE(((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0,
             "ft_conv_embed: pointers must be 16-byte aligned");
  const int Cv = C * elt_bytes / 16;
  const long long total = static_cast<long long>(planes) * N * Hp * Wp * Cv;
  conv_embed_kernel<<<layout_grid(total, device), 256, 0, stream>>>(
      static_cast<const uint4*>(src), static_cast<uint4*>(dst), N, H, W, Cv, Hp, Wp, oh, ow, planes);
  FT_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return FT_E_OK;
}

// src [N, Hp, Wp, C] -> dst [N, Ho, Wo, C]: dst[n, i, j] = src[n, i + oh, j + ow].
FT_API int ft_conv_crop(const void* src, void* dst, int N, int Ho, int Wo, int C, int Hp, int Wp, int oh, int ow,
                        int elt_bytes, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  FT_REQUIRE(src && dst, "ft_conv_crop: null pointer");
  FT_REQUIRE(N > 0 && Ho > 0 && Wo > 0 && C > 0 && oh >= 0 && ow >= 0 && Ho + oh <= Hp && Wo + ow <= Wp,
             "ft_conv_crop: the window does not fit the source grid");
  FT_REQUIRE((elt_bytes == 2 || elt_bytes == 4) && (C * elt_bytes) % 16 == 0,
             "ft_conv_crop: a pixel (%d channels x %d bytes) must be a multiple of 16 bytes", C, elt_bytes);
  FT_REQUIRE(((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0,
             "ft_conv_crop: pointers must be 16-byte aligned");
  const int Cv = C * elt_bytes / 16;
  const long long total = static_cast<long long>(N) * Ho * Wo * Cv;
  conv_crop_kernel<<<layout_grid(total, device), 256, 0, stream>>>(
      static_cast<const uint4*>(src), static_cast<uint4*>(dst), N, Ho, Wo, Cv, Hp, Wp, oh, ow);
  FT_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return FT_E_OK;
}

// x [N, H, W, C] bf16 -> out [N*Ho*Wo, Kpad] bf16 patches (Kpad >= KH*KW*C, Kpad % 8 == 0).
FT_API int ft_im2col_nhwc(const void* x, void* out, int N, int H, int W, int C, int KH, int KW, int stride,
                          int ph, int pw, int dil, int Kpad, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  FT_REQUIRE(x && out, "ft_im2col_nhwc: null pointer");
  FT_REQUIRE(N > 0 && H > 0 && W > 0 && C > 0 && KH > 0 && KW > 0 && stride > 0 && dil > 0 && ph >= 0 && pw >= 0,
             "ft_im2col_nhwc: bad geometry");
  const int eh = H + 2 * ph - dil * (KH - 1) - 1, ew = W + 2 * pw - dil * (KW - 1) - 1;
  FT_REQUIRE(eh >= 0 && ew >= 0, "ft_im2col_nhwc: the filter does not fit the padded input");
  FT_REQUIRE(Kpad >= KH * KW * C && Kpad % 8 == 0, "ft_im2col_nhwc: Kpad=%d too small or not a multiple of 8", Kpad);
  const int Ho = eh / stride + 1, Wo = ew / stride + 1;
  const long long total = static_cast<long long>(N) * Ho * Wo * (KH * KW + 1);
  if (C == 4 && Kpad % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) & 7) | (reinterpret_cast<uintptr_t>(out) & 15)) == 0 &&
      static_cast<long long>(N) * Ho * Wo < (1ll << 31) - (1 << 20) && static_cast<long long>(H) * W < (1ll << 31)) {
    im2col_c4_kernel<<<sm_count(device) * 8, 256, 0, stream>>>(static_cast<const uint2*>(x), static_cast<uint4*>(out), N, H, W, KH, KW, stride,
                                                               ph, pw, dil, Ho, Wo, Kpad / 8);
    FT_CUDA_CHECK(cudaGetLastError());
    count_launch();
    return FT_E_OK;
  }
  im2col_nhwc_kernel<<<layout_grid(total, device), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(out), N, H, W, C, KH, KW, stride, ph, pw,
      dil, Ho, Wo, Kpad);
  FT_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return FT_E_OK;
}

// dst (+)= src over n0 x n1 x n2 elements with their own strides (elements); *_f32: fp32 instead of bf16; order (or null): n[order_dim]
// places of src along that dimension, at most 64.
FT_API int ft_filter_copy(const void* src, void* dst, const int* n, const long long* src_strides, const long long* dst_strides, int src_f32,
                          int dst_f32, int accumulate, int order_dim, const int* order, int device, cudaStream_t stream) {
  if (int _rc = ft::ensure_device(device)) return _rc;
  FT_REQUIRE(src && dst && n && src_strides && dst_strides, "ft_filter_copy: null pointer");
  FilterCopy f{};
  long long total = 1;
  for (int k = 0; k < 3; ++k) {
    FT_REQUIRE(n[k] > 0, "ft_filter_copy: empty dimension");
    f.n[k] = n[k]; f.ss[k] = src_strides[k]; f.ds[k] = dst_strides[k];
    total *= n[k];
  }
  FT_REQUIRE(total < (1ll << 31) - (1 << 22), "ft_filter_copy: too many elements");
  f.src_f32 = src_f32; f.dst_f32 = dst_f32; f.accumulate = accumulate; f.order_dim = -1;
  if (order) {
    FT_REQUIRE(order_dim >= 0 && order_dim < 3 && n[order_dim] <= 64, "ft_filter_copy: bad order");
    f.order_dim = order_dim;
    for (int i = 0; i < n[order_dim]; ++i) f.order[i] = static_cast<unsigned char>(order[i]);
  }
  filter_copy_kernel<<<layout_grid(total, device), 256, 0, stream>>>(src, dst, f);
  FT_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return FT_E_OK;
}
