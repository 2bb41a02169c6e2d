// Inverse FFT of lines held in shared memory, for the image passes of the
// objective (objective.cu) and of the gradient (dchi2_nu.cu): radix-8
// Stockham passes with the butterflies in registers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gv {

// The arithmetic that more than one kernel performs on the same values (the
// FFT butterflies and twiddles, the phase rotation, the degridding's model
// and chi2 terms, the prior stencils) spells out every multiply-add with
// rounding intrinsics: the compiler never contracts those, so the separate
// kernels and the fused ones round each operation alike wherever the code
// is inlined (the compiler's choice of which product to fuse into an FMA
// can otherwise differ between inlining contexts).
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                     __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}

// R-point inverse DFT (exp(+2 pi i r s / R), R = 2^LR <= 8) of v in
// registers, radix-2 decimation in frequency: the result is in bit-reversed
// order (X[r] = v[brev(r)]).  The twiddles are 1, i and (+-1 + i)/sqrt(2):
// multiplications by 1 and i are exact.
__device__ __forceinline__ float2 rot_turn(float2 d, int s, int m) {
  // d * e^{2 pi i s / m}, m in {2, 4, 8}, s < m / 2 (compile-time after
  // unrolling)
  const float c = 0.70710678118654752440f;
  if (s == 0) return d;
  if (m == 4 || s == 2) return make_float2(-d.y, d.x);                 // * i
  if (s == 1) return make_float2(__fmul_rn(c, d.x - d.y), __fmul_rn(c, d.x + d.y));  // * (1 + i)/sqrt 2
  return make_float2(__fmul_rn(c, -d.x - d.y), __fmul_rn(c, d.x - d.y));           // * (-1 + i)/sqrt 2
}

template <int LR>
__device__ __forceinline__ void dft_inv(float2 (&v)[1 << LR]) {
  constexpr int R = 1 << LR;
#pragma unroll
  for (int half = R / 2; half >= 1; half >>= 1) {
#pragma unroll
    for (int g = 0; g < R; g += 2 * half) {
#pragma unroll
      for (int s = 0; s < half; s++) {
        const float2 a = v[g + s], b = v[g + s + half];
        v[g + s] = make_float2(a.x + b.x, a.y + b.y);
        v[g + s + half] = rot_turn(make_float2(a.x - b.x, a.y - b.y), s, 2 * half);
      }
    }
  }
}

template <int LR>
__device__ __forceinline__ constexpr int brev_c(int r) {
  int o = 0;
  for (int b = 0; b < LR; b++) o |= ((r >> b) & 1) << (LR - 1 - b);
  return o;
}

// Shared-memory position of element e of an FFT line: one float2 of padding
// after every eight, so the first Stockham pass's writes (eight elements
// apart across the lanes) and the second's (runs of eight, 64 apart) fall in
// distinct banks.  A line of n elements takes fft_span(n) positions; the
// lines of a multi-column buffer are fft_stride(n) apart (four more, so four
// columns read row by row do not share banks either).
__device__ __forceinline__ int fpad(int e) { return e + (e >> 3); }
__host__ __device__ constexpr int fft_span(int n) { return n + (n >> 3); }
__host__ __device__ __forceinline__ int fft_stride(int n) { return fft_span(n) + 4; }

// One Stockham autosort pass of radix R = 2^LR over `ncol` columns of length
// n = 2^log2n in shared memory (element e of column c at
// buf[c * fft_stride(n) + fpad(e)], natural order).
// Work item (c, j), j < n / R, reads x[j + r n/R] (r < R), multiplies by the
// twiddles e^{2 pi i r k / (Ns R)} with k = j mod Ns (table tw[m] =
// e^{2 pi i m / n}, read through L1), takes the R-point inverse DFT and
// writes y[(j / Ns) Ns R + k + r Ns] (Govindaraju et al., "High Performance
// Discrete Fourier Transforms on Graphics Processors", SC 2008).  In place:
// all items are read before a block barrier and written after it, so each
// thread holds its items' values in registers: max(VPT, R) of them, VPT the
// values per thread (ncol * n <= VPT * blockDim.x).
template <int LR, int VPT>
__device__ __forceinline__ void stockham_pass(float2* buf, int log2n, int ncol, int lNs,
                                              const float2* __restrict__ tw) {
  constexpr int R = 1 << LR;
  constexpr int kMaxItems = VPT / R > 1 ? VPT / R : 1;
  const int lq = log2n - LR;  // log2 of the items per column
  const int items = ncol << lq;
  float2 v[kMaxItems][R];
#pragma unroll
  for (int t = 0; t < kMaxItems; t++) {
    const int it = threadIdx.x + t * blockDim.x;
    if (it < items) {
      const int c = it >> lq, j = it & ((1 << lq) - 1);
      const float2* x = buf + c * fft_stride(1 << log2n);
#pragma unroll
      for (int r = 0; r < R; r++) v[t][r] = x[fpad(j + (r << lq))];
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < kMaxItems; t++) {
    const int it = threadIdx.x + t * blockDim.x;
    if (it < items) {
      const int c = it >> lq, j = it & ((1 << lq) - 1);
      const int k = j & ((1 << lNs) - 1);
      if (lNs > 0) {
        const int step = k << (log2n - lNs - LR);  // r k n / (Ns R) = r * step
#pragma unroll
        for (int r = 1; r < R; r++) v[t][r] = cmul(v[t][r], __ldg(tw + r * step));
      }
      dft_inv<LR>(v[t]);
      float2* y = buf + c * fft_stride(1 << log2n);
      const int base = ((j >> lNs) << (lNs + LR)) + k;
#pragma unroll
      for (int r = 0; r < R; r++) y[fpad(base + (r << lNs))] = v[t][brev_c<LR>(r)];
    }
  }
  __syncthreads();
}

// In-place inverse FFT (cuFFT's CUFFT_INVERSE convention: exp(+i),
// unnormalised) of `ncol` independent columns of length n = 2^log2n held in
// shared memory (element e of column c at buf[c * fft_stride(n) + fpad(e)]),
// natural order in and out: radix-8
// Stockham passes, then one of radix 4 or 2.  The caller has synchronised
// the block after filling buf; needs ncol * n <= VPT * blockDim.x and
// n <= 2 * blockDim.x * max(1, VPT / 2).
template <int VPT>
__device__ void smem_fft(float2* buf, int log2n, int ncol, const float2* __restrict__ tw) {
  int lNs = 0;
  while (log2n - lNs >= 3) {
    stockham_pass<3, VPT>(buf, log2n, ncol, lNs, tw);
    lNs += 3;
  }
  if (log2n - lNs == 2) stockham_pass<2, VPT>(buf, log2n, ncol, lNs, tw);
  else if (log2n - lNs == 1) stockham_pass<1, VPT>(buf, log2n, ncol, lNs, tw);
}

// ---- 8 values a thread, the passes above ------------------------------------
// The same transform as smem_fft (the same butterflies and twiddles on the
// same values, so the same bits) of a line of n = 2^LG elements by n / 8
// threads, thread j holding elements j + e n / 8 (e < 8) in v before the first
// pass and after the last, in natural order of e.  The first pass takes its
// elements from the caller's registers and the last leaves them there, so a
// 2048-point line crosses shared memory three times instead of five, with 6
// barriers instead of 10; the twiddles lie pass by pass in lane order (a
// strided table costs a sector per lane).  `buf` holds fft_span(2^LG) float2.
//
// Table: for every pass after the first, with Ns the product of the radices
// before it and R its radix, e^{2 pi i r k / (R Ns)} at (r - 1) Ns + k,
// 1 <= r < R, k < Ns.
__host__ __device__ constexpr int fft8_radix(int lg, int l) { return lg - l >= 3 ? 3 : lg - l; }
__host__ __device__ constexpr int fft8_twiddles(int lg) {
  int n = 0;
  for (int l = 3; l < lg; l += 3) n += ((1 << fft8_radix(lg, l)) - 1) << l;
  return n;
}

template <int LG, int L>
__device__ __forceinline__ void fft8_passes(float2 (&v)[8], float2* buf, int j,
                                            const float2* __restrict__ tw) {
  constexpr int T = (1 << LG) / 8, LR = fft8_radix(LG, L), R = 1 << LR, M = 8 / R;
  // the last pass' results: element ((j >> L - 3) << L) + k + r 2^(L - 3),
  // then elements j + e T of the next.  Each exchange has the padding that
  // puts the writes of a half warp into distinct banks and leaves the reads of
  // 16 neighbours together: one position in 16 after the first pass (writes 8
  // apart), 8 in 64 after the second (runs of 8, 64 apart), none after that.
  // (One in 8 throughout made every read a bank conflict; the row pass runs
  // its data pipe at three quarters of its rate.)
  const int kw = j & ((1 << (L - 3)) - 1), base = ((j >> (L - 3)) << L) + kw;
  auto place = [](int e) { return L == 3 ? e + (e >> 4) : (L == 6 ? e + 8 * (e >> 6) : e); };
  constexpr int kStep = 1 << (L - 3);
  // base + r kStep stays in base's group of the padding
  float2* y = buf + place(base);
#pragma unroll
  for (int r = 0; r < 8; r++) y[r * kStep] = v[brev_c<3>(r)];
  __syncthreads();
  constexpr int kGroup = L == 3 ? 16 : (L == 6 ? 64 : 1);
#pragma unroll
  for (int e = 0; e < 8; e++)
    v[e] = T % kGroup == 0 ? buf[place(j) + e * place(T)] : buf[place(j + e * T)];
  if constexpr (LR == 3) {
    const int k = j & ((1 << L) - 1);
#pragma unroll
    for (int r = 1; r < 8; r++) v[r] = cmul(v[r], __ldg(tw + ((r - 1) << L) + k));
    dft_inv<3>(v);
    if constexpr (L + 3 < LG) {
      __syncthreads();
      fft8_passes<LG, L + 3>(v, buf, j, tw + (7 << L));
    } else {
      float2 u[8];
#pragma unroll
      for (int r = 0; r < 8; r++) u[r] = v[brev_c<3>(r)];
#pragma unroll
      for (int r = 0; r < 8; r++) v[r] = u[r];
    }
  } else {
#pragma unroll
    for (int m = 0; m < M; m++) {
      float2 u[R];
      u[0] = v[m];
#pragma unroll
      for (int r = 1; r < R; r++) u[r] = cmul(v[m + r * M], __ldg(tw + ((r - 1) << L) + j + m * T));
      dft_inv<LR>(u);
#pragma unroll
      for (int r = 0; r < R; r++) v[m + r * M] = u[brev_c<LR>(r)];
    }
  }
}

template <int LG>
__device__ __forceinline__ void fft8(float2 (&v)[8], float2* buf, int j,
                                     const float2* __restrict__ tw) {
  dft_inv<3>(v);
  fft8_passes<LG, 3>(v, buf, j, tw);
}

// ---- 16 values a thread, radix 16 -----------------------------------------
// Inverse FFT of a line of n = 2^LG elements by n / 16 threads, thread j
// holding elements j + e n / 16 (e < 16) in v before and after every pass: a
// first pass of radix 2^((LG - 1) % 4 + 1), then radix 16.  Against the
// radix-8 passes above: the first pass reads its elements from where the
// caller has them and the last leaves them in registers, so a 4096-point line
// crosses shared memory twice instead of five times, with 4 barriers instead
// of 10; the twiddles lie pass by pass in the order the lanes read them.
//
// Shared-memory position of element e: one float2 of padding after every 16,
// which puts every write and read of a half warp into distinct banks.
__device__ __forceinline__ int pad16(int e) { return e + (e >> 4); }
__host__ __device__ constexpr int span16(int n) { return n + (n >> 4); }

// multiplication by e^{2 pi i s / 16}, 0 <= s < 8 (compile-time after unrolling)
__device__ __forceinline__ float2 rot16(float2 d, int s) {
  constexpr float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
  if (s == 1) return cmul(d, make_float2(c1, s1));
  if (s == 3) return cmul(d, make_float2(s1, c1));
  if (s == 5) return cmul(d, make_float2(-s1, c1));
  if (s == 7) return cmul(d, make_float2(-c1, s1));
  return rot_turn(d, s >> 1, 8);
}

// 16-point inverse DFT in registers; X[r] = v[brev_c<4>(r)]
__device__ __forceinline__ void dft16(float2 (&v)[16]) {
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const float2 a = v[s], b = v[s + 8];
    v[s] = make_float2(a.x + b.x, a.y + b.y);
    v[s + 8] = rot16(make_float2(a.x - b.x, a.y - b.y), s);
  }
  float2(&lo)[8] = reinterpret_cast<float2(&)[8]>(v[0]);
  float2(&hi)[8] = reinterpret_cast<float2(&)[8]>(v[8]);
  dft_inv<3>(lo);
  dft_inv<3>(hi);
}

__host__ __device__ constexpr int fft16_first(int lg) { return (lg - 1) % 4 + 1; }

// Entries of the twiddle table of a 2^lg-point line: for every pass after the
// first, with Ns = the product of the radices before it,
// e^{2 pi i r k / (16 Ns)} at (r - 1) Ns + k, 1 <= r < 16, k < Ns.
__host__ __device__ constexpr int fft16_twiddles(int lg) {
  int n = 0;
  for (int l = fft16_first(lg); l < lg; l += 4) n += 15 << l;
  return n;
}

// All passes of a line; `buf` holds span16(2^LG) float2 for it, and every
// thread of the block makes the same calls.  On return element x of the
// result with x = j + r n / 16 is v[brev_c<4>(r)].
template <int LG>
__device__ __forceinline__ void fft16(float2 (&v)[16], float2* buf, int j,
                                      const float2* __restrict__ tw) {
  constexpr int T = (1 << LG) / 16, L0 = fft16_first(LG), R0 = 1 << L0, M0 = 16 / R0;
  if constexpr (L0 == 4) {
    dft16(v);
  } else {
#pragma unroll
    for (int m = 0; m < M0; m++) {
      float2 u[R0];
#pragma unroll
      for (int r = 0; r < R0; r++) u[r] = v[m + r * M0];
      dft_inv<L0>(u);
#pragma unroll
      for (int r = 0; r < R0; r++) v[m + r * M0] = u[r];
    }
  }
  // y[R0 (j + m T) + r] of item m.  Written as one padded position and
  // constants (r < R0 never carries into the padding's multiple of 16), here
  // and below: the compiler does not see through the shift
  constexpr bool kWide = (R0 * T) % 16 == 0;
  {
    float2* y = buf + pad16(R0 * j);
#pragma unroll
    for (int m = 0; m < M0; m++)
#pragma unroll
      for (int r = 0; r < R0; r++) {
        const float2 x = v[m + brev_c<L0>(r) * M0];
        if constexpr (kWide) y[m * span16(R0 * T) + r] = x;
        else buf[pad16(R0 * (j + m * T) + r)] = x;
      }
  }
#pragma unroll
  for (int l = L0; l < LG; l += 4) {
    const int k = j & ((1 << l) - 1);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 16; r++)
      v[r] = T % 16 == 0 ? buf[pad16(j) + r * span16(T)] : buf[pad16(j + r * T)];
#pragma unroll
    for (int r = 1; r < 16; r++) v[r] = cmul(v[r], __ldg(tw + ((r - 1) << l) + k));
    tw += 15 << l;
    dft16(v);
    if (l + 4 < LG) {
      __syncthreads();
      float2* y = buf + pad16(((j >> l) << (l + 4)) + k);
#pragma unroll
      for (int r = 0; r < 16; r++) y[(r << l) + ((r << l) >> 4)] = v[brev_c<4>(r)];
    }
  }
}

}  // namespace gv
