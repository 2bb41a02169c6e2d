// Operands of the convolution GEMMs (k_gemm, cnn.cu): where the elements of the
// three products lie in the tensors.  A tensor may hold 2^31 elements and more
// (the 48-channel concatenation of a 2048^2 network at batch 11), so offsets
// are 64 bits wide; a batch's pixels and a side's stay in 32.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gv {
namespace cnn {

// A channel slice of an NCHW tensor: element (b, c, y, x) of the slice is
// p[((b * C + c0 + c) * H + y) * W + x].
struct View {
  float* p;
  int C, c0;
};

__device__ __host__ inline bool rows_of_eight(const float* p, int W) {
  return W % 8 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

// A pixel of an operand: its offset in the first channel, row, column, batch.
struct Pixel {
  int64_t off;
  int y, x, b;
};
// A row of a result: its number and the offset of its pixel in channel 0.
struct OutRow {
  int m;
  int64_t off;
};

// forward: y = act(conv(x) + bias); with split-K (part set) each split
// stores its partial sum to part[split][n][m] and k_conv_fwd_finish adds
// the splits, the bias and the activation
struct ConvFwdOp {
  static constexpr bool kPixelRows = true;
  static constexpr bool kFlip = false;
  const float* x;
  int xC, xc0;
  const float* w;
  const uint4* packed;  // BF16 tile images of w (k_pack_weights), or null
  const float* bias;
  float* y;
  int yC, yc0;
  int Cin, Cout, H, W, ks, relu;
  float* part;
  int M;
  bool fast;
  __device__ const float* src() const { return x; }
  __host__ __device__ Pixel pixel(int m) const {
    const int HW = H * W;
    const int b = m / HW, r = m - b * HW, y0 = r / W;
    return {(int64_t)(b * xC + xc0) * HW + r, y0, r - y0 * W, b};
  }
  __device__ float a(int m, int k) const {
    const int HW = H * W;
    const int b = m / HW, r = m - b * HW, y0 = r / W, x0 = r - y0 * W;
    const int kk = ks * ks, cin = k / kk, t = k - cin * kk;
    const int yy = y0 + t / ks - ks / 2, xx = x0 + t % ks - ks / 2;
    if ((unsigned)yy >= (unsigned)H || (unsigned)xx >= (unsigned)W) return 0.0f;
    return x[((size_t)(b * xC + xc0 + cin) * H + yy) * W + xx];
  }
  __device__ float b(int k, int n) const { return w[(size_t)n * Cin * ks * ks + k]; }
  __device__ const float* grad_row(int, const Pixel&) const { return nullptr; }
  __host__ __device__ OutRow row(int m) const {
    const int HW = H * W;
    const int b = m / HW, r = m - b * HW;
    return {m, (int64_t)(b * yC + yc0) * HW + r};
  }
  __device__ void store(const OutRow& at, int n, int cnt, float (&v)[8], int split) const {
    float* out = part ? part + ((size_t)split * Cout + n) * M + at.m
                      : y + at.off + (size_t)n * H * W;
    const size_t step = part ? (size_t)M : (size_t)H * W;
    if (!part) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (j < cnt) v[j] += __ldg(bias + n + j);
        if (relu) v[j] = fmaxf(v[j], 0.0f);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j < cnt) out[j * step] = v[j];
  }
};

// backward data: dx = conv of dz with the taps flipped; with `act` (the
// activation whose gradient dx is) masked by its ReLU
struct ConvBwdDataOp {
  static constexpr bool kPixelRows = true;
  static constexpr bool kFlip = true;  // the taps run backwards
  const float* dz;
  int zC, zc0;
  const float* w;
  const uint4* packed;
  float* dx;
  int xC, xc0;
  const float* act;
  int aC, ac0;
  int Cin, Cout, H, W, ks;
  bool fast;
  __device__ const float* src() const { return dz; }
  __host__ __device__ Pixel pixel(int m) const {
    const int HW = H * W;
    const int b = m / HW, r = m - b * HW, y0 = r / W;
    return {(int64_t)(b * zC + zc0) * HW + r, y0, r - y0 * W, b};
  }
  __device__ float a(int m, int k) const {
    const int HW = H * W;
    const int b = m / HW, r = m - b * HW, y0 = r / W, x0 = r - y0 * W;
    const int kk = ks * ks, co = k / kk, t = k - co * kk;
    const int yy = y0 - t / ks + ks / 2, xx = x0 - t % ks + ks / 2;
    if ((unsigned)yy >= (unsigned)H || (unsigned)xx >= (unsigned)W) return 0.0f;
    return dz[((size_t)(b * zC + zc0 + co) * H + yy) * W + xx];
  }
  __device__ float b(int k, int n) const {
    const int kk = ks * ks, co = k / kk, t = k - co * kk;
    return w[((size_t)co * Cin + n) * kk + t];
  }
  __device__ const float* grad_row(int, const Pixel&) const { return nullptr; }
  __device__ int2 row(int m) const {
    const int HW = H * W;
    const int b = m / HW;
    return make_int2(b, m - b * HW);
  }
  __device__ void store(const int2& at, int n, int cnt, float (&v)[8], int) const {
    const int HW = H * W;
    if (act) {
      const float* a = act + (size_t)(at.x * aC + ac0 + n) * HW + at.y;
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (j < cnt && !(__ldg(a + (size_t)j * HW) > 0.0f)) v[j] = 0.0f;
    }
    float* out = dx + (size_t)(at.x * xC + xc0 + n) * HW + at.y;
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j < cnt) out[(size_t)j * HW] = v[j];
  }
};

// backward weight: partial[split][cout][cin*ks*ks] = sum over this split's
// pixels of dz * x (shifted)
struct ConvBwdWeightOp {
  static constexpr bool kPixelRows = false;
  static constexpr bool kFlip = false;
  const float* x;
  int xC, xc0;
  const float* dz;
  int zC, zc0;
  float* partial;
  int Cin, Cout, H, W, ks;
  bool fast;
  static constexpr const uint4* packed = nullptr;
  __device__ const float* src() const { return x; }
  __host__ __device__ Pixel pixel(int k) const {
    const int HW = H * W;
    const int b = k / HW, r = k - b * HW, y0 = r / W;
    return {(int64_t)(b * xC + xc0) * HW + r, y0, r - y0 * W, b};
  }
  __device__ float a(int m, int k) const {
    const int kk = ks * ks, cin = m / kk, t = m - cin * kk;
    const int HW = H * W;
    const int b = k / HW, r = k - b * HW, y0 = r / W, x0 = r - y0 * W;
    const int yy = y0 + t / ks - ks / 2, xx = x0 + t % ks - ks / 2;
    if ((unsigned)yy >= (unsigned)H || (unsigned)xx >= (unsigned)W) return 0.0f;
    return x[((size_t)(b * xC + xc0 + cin) * H + yy) * W + xx];
  }
  __device__ float b(int k, int n) const {
    const int HW = H * W;
    const int b = k / HW, r = k - b * HW;
    return dz[(size_t)(b * zC + zc0 + n) * HW + r];
  }
  __device__ const float* grad_row(int n, const Pixel& p) const {
    return dz + (size_t)(p.b * zC + zc0 + n) * H * W + p.y * W + p.x;
  }
  __device__ int row(int m) const { return m; }
  __device__ void store(int m, int n, int cnt, float (&v)[8], int split) const {
    const size_t row = (size_t)Cin * ks * ks;
    float* out = partial + split * Cout * row + n * row + m;
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (j < cnt) out[j * row] = v[j];
  }
};

}  // namespace cnn
}  // namespace gv
