// Warm-start network: a 2-D U-Net (encoder-decoder with skip connections)
// trained on (dirty image + PSF, converged image) pairs.  No counterpart in
// the reference; it is the learned part of the imaging objective path.
//
// Every convolution, in the forward pass and in both backward passes, is a
// BF16 GEMM on the tcgen05 tensor cores with FP32 accumulation in TMEM
// (k_gemm below):
//   forward      M = B*H*W pixels, N = Cout, K = Cin*ks*ks
//   bwd data     M = B*H*W pixels, N = Cin,  K = Cout*ks*ks (flipped taps)
//   bwd weight   M = Cin*ks*ks,    N = Cout, K = B*H*W (split over K, the
//                splits summed in a fixed order)
// The operand tiles are staged by the CTA's threads straight from the FP32
// NCHW activations (im2col on the fly, rounded to BF16) into 128-byte
// swizzled shared-memory tiles; one thread issues the MMAs; two stages
// alternate, the next chunk's loads under way.  The epilogue (bias, ReLU,
// layout) is applied on the way out of TMEM.  Pooling, upsampling, the loss
// and Adam are plain bandwidth-bound kernels.
//
// Layout of the network (levels l = 0..L-1, C_l = c0 * 2^l channels, side
// H / 2^l):  enc_l = relu(conv(relu(conv(in_l)))), in_{l+1} = avgpool2(enc_l);
// dec_{L-1} = enc_{L-1}; dec_l = relu(conv(relu(conv([up2(dec_{l+1}), enc_l]))));
// out = conv1x1(dec_0).  Parameters are one flat FP32 vector, layer by layer
// (weights [Cout][Cin][ks][ks], then bias [Cout]) in the order enc_0 ..
// enc_{L-1}, dec_{L-2} .. dec_0, out.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include "conv_ops.cuh"
#include "gv_internal.cuh"
#include "tcgen05.cuh"

namespace gv {
namespace cnn {

using namespace gv::tc;

// ---------------------------------------------------------------- GEMM core
// 11 warps: with 3 x 3 taps the eight-pixel groups of an A tile are 352 loads
constexpr int kBM = 128, kBK = 64, kGemmThreads = 352;

__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <int BN>
struct GemmLayout {
  static constexpr uint32_t kSboA = (kBM / 64) * 1024;
  static constexpr uint32_t kTileA = kSboA * (kBK / 8);
  static constexpr uint32_t kSboB = (BN / 64) * 1024;
  static constexpr uint32_t kTileB = kSboB * (kBK / 8);
  static constexpr uint32_t kStage = kTileA + kTileB;
  static constexpr uint32_t kSmem = 1024 + 2 * kStage;
};

// byte offset of the 16-byte chunk holding columns 8*g..8*g+7 of row r in a
// K-major 128B-swizzled tile (64 columns a row, atoms of 8 rows 1024 B apart)
__device__ __forceinline__ uint32_t kmajor_off(int r, int g) {
  return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((g ^ (r & 7)) << 4));
}

__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(bf16x2(v[0], v[1]), bf16x2(v[2], v[3]), bf16x2(v[4], v[5]),
                    bf16x2(v[6], v[7]));
}

// Eight pixels of an image row (16-byte aligned) and the ones beside them.
struct Row {
  float4 a, b;
  float l, r;  // zero outside the row
  __device__ __forceinline__ void clear() {
    a = b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    l = r = 0.0f;
  }
  template <bool kEnds>
  __device__ __forceinline__ void load(const float* __restrict__ p, int x, int W) {
    a = __ldg(reinterpret_cast<const float4*>(p));
    b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    if (kEnds) {
      l = x > 0 ? __ldg(p - 1) : 0.0f;
      r = x + 8 < W ? __ldg(p + 8) : 0.0f;
    }
  }
  __device__ __forceinline__ uint4 centre() const {
    return make_uint4(bf16x2(a.x, a.y), bf16x2(a.z, a.w), bf16x2(b.x, b.y), bf16x2(b.z, b.w));
  }
  // the row one to the left, as it is and one to the right
  __device__ __forceinline__ void shifted(uint4 (&v)[3]) const {
    const uint32_t w1 = bf16x2(a.y, a.z), w2 = bf16x2(a.w, b.x), w3 = bf16x2(b.y, b.z);
    v[0] = make_uint4(bf16x2(l, a.x), w1, w2, w3);
    v[1] = centre();
    v[2] = make_uint4(w1, w2, w3, bf16x2(b.w, r));
  }
};

// D[m][n] = sum_k A[m][k] B[k][n] over this CTA's K range; op.a(m,k),
// op.b(k,n) fetch FP32 operands, op.store(row, n, count, v, split) writes up to
// eight columns of a result.
//
// KS (3 or 1: the taps of a row; tensors aligned, rows multiples of eight
// pixels) stages the tiles in groups of eight pixels; KS = 0 element by
// element.  What bounds the network's GEMMs is the way from one chunk of 64 k
// to the next (few chunks or few CTAs each, MMAs of well under a microsecond),
// so a chunk's loads are issued before the last one's MMAs, into registers,
// and cost little:
//   A  a row of the tile is a channel and a tap.  The three taps of an image
//      row are one load of the group and its two neighbours, rounded once and
//      stored three times: 22 such units x 16 groups where the rows are k
//      (Op::kPixelRows: forward, data gradient; MN-major), 44 x 8 where they
//      are m (weight gradient; K-major), one a thread.  Neighbouring threads
//      take neighbouring groups: with a row a thread, as this was first, each
//      load of the weight gradient touched 32 lines.
//   B  the weights as ready BF16 tile images (op.packed), or the gradient.
// Bound by the instructions (two thirds of the issue slots at
// the shallow levels).  The network of 256^2, 16 channels, 5 levels, with this
// staging, the epilogue's eight columns and the narrower tiles: a training step
// of batch 8 5310 -> 2670 us, a forward pass of one sky 342 -> 224.  One CTA
// for several row tiles, with the next one's loads under the last one's
// epilogue, gave nothing (236 -> 244).
template <class Op, int BN, int KS>
__global__ void __launch_bounds__(kGemmThreads, Op::kPixelRows && BN == 64 ? 3 : (BN < 256 ? 2 : 1))
    k_gemm(Op op, int M, int N, int K, int klen, uint32_t* err) {
  using L = GemmLayout<BN>;
  constexpr int T = kGemmThreads;
  constexpr bool kRows = Op::kPixelRows;
  constexpr bool kmajor = !kRows && KS > 0;
  constexpr int kGroups = kRows ? kBM / 8 : kBK / 8;  // of eight pixels
  constexpr int kRowsA = kRows ? kBK : kBM;
  constexpr int kUnits = KS == 3 ? (kRowsA + 4) / 3 : kRowsA;
  constexpr int kLoadsA = KS > 0 ? (kUnits * kGroups + T - 1) / T : 1;
  constexpr int kLoadsB = KS == 0 ? 1 : kRows ? ((int)(L::kTileB / 16) + T - 1) / T
                                              : (BN * kGroups + T - 1) / T;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* base = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  __shared__ uint64_t bar[2];
  __shared__ uint32_t tslot;
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
  const int kbeg = blockIdx.z * klen;
  const int kend = min(K, kbeg + klen);
  const int nch = kend > kbeg ? (kend - kbeg + kBK - 1) / kBK : 0;

  const int grp = tid % kGroups;  // T is a multiple of both
  Pixel at{0, 0, 0, 0};             // the group's first
  const int mg = m0 + grp * 8;
  if (KS > 0 && kRows && mg < M) at = op.pixel(mg);  // M is a multiple of eight
  // the first unit that touches the tile's rows from row0 on
  auto unit = [&](int row0, int i) {
    return (KS == 3 ? row0 / 3 : row0) + (tid + i * T) / kGroups;
  };
  // B's tile images: 64 columns each, the 8-row atoms of a wider tile side by side
  constexpr int kAtoms = BN / 64, kImage = kBK * 64 / 8;  // uint4 of an image
  auto image = [&](int c, int e) {
    const int atom = e >> 6;
    return op.packed + ((size_t)(blockIdx.y * kAtoms + atom % kAtoms) * ((K + kBK - 1) / kBK) +
                        (kbeg / kBK + c)) * kImage + (atom / kAtoms) * 64 + (e & 63);
  };
  Row ra[kLoadsA];
  Row rb[kmajor ? kLoadsB : 1];
  uint4 rw[kRows ? kLoadsB : 1];
  auto load = [&](int c) {
    const int k0 = kbeg + c * kBK;
    const int rows = kRows ? K : M;
    const bool in = kRows ? mg < M : k0 + 8 * grp < kend;
    if (!kRows && in) at = op.pixel(k0 + 8 * grp);
#pragma unroll
    for (int i = 0; i < kLoadsA; i++) {
      ra[i].clear();
      const int u = unit(kRows ? k0 : m0, i), ch = KS == 3 ? u / 3 : u;
      int dy = KS == 3 ? u - 3 * ch - 1 : 0;
      if (Op::kFlip) dy = -dy;
      if (in && tid + i * T < kUnits * kGroups && u * max(KS, 1) < rows &&
          (unsigned)(at.y + dy) < (unsigned)op.H)
        ra[i].template load<KS == 3>(op.src() + at.off + (int64_t)ch * (op.H * op.W) + dy * op.W,
                                     at.x, op.W);
    }
    if constexpr (kmajor) {
#pragma unroll
      for (int i = 0; i < kLoadsB; i++) {
        rb[i].clear();
        const int r = (tid + i * T) / kGroups;
        if (in && r < BN && n0 + r < N)
          rb[i].template load<false>(op.grad_row(n0 + r, at), at.x, op.W);
      }
    } else if (kRows) {
      if (op.packed) {
#pragma unroll
        for (int i = 0; i < kLoadsB; i++)
          if (tid + i * T < (int)(L::kTileB / 16)) rw[i] = __ldg(image(c, tid + i * T));
      }
    }
  };
  auto put = [&](int c, uint8_t* sa, uint8_t* sb) {
    const int row0 = kRows ? kbeg + c * kBK : m0;
#pragma unroll
    for (int i = 0; i < kLoadsA; i++) {
      if (tid + i * T >= kUnits * kGroups) break;
      uint4 v[3];
      if (KS == 3) ra[i].shifted(v);
      else v[0] = ra[i].centre();
      const int r0 = unit(row0, i) * KS - row0;
#pragma unroll
      for (int j = 0; j < KS; j++) {
        const int r = r0 + j;
        if (r < 0 || r >= kRowsA) continue;
        const uint32_t off = kRows ? tile_off(grp >> 3, grp & 7, r, L::kSboA) : kmajor_off(r, grp);
        *reinterpret_cast<uint4*>(sa + off) = v[Op::kFlip && KS == 3 ? 2 - j : j];
      }
    }
    if constexpr (kmajor) {
#pragma unroll
      for (int i = 0; i < kLoadsB; i++) {
        const int r = (tid + i * T) / kGroups;
        // beyond the last column: zeros, once in each stage
        if (r < BN && (n0 + r < N || c < 2))
          *reinterpret_cast<uint4*>(sb + kmajor_off(r, grp)) = rb[i].centre();
      }
    } else if (kRows) {
      if (op.packed) {
#pragma unroll
        for (int i = 0; i < kLoadsB; i++)
          if (tid + i * T < (int)(L::kTileB / 16))
            reinterpret_cast<uint4*>(sb)[tid + i * T] = rw[i];
      }
    }
  };
  if (KS > 0 && nch > 0) load(0);

  if (warp == 0) {
    tmem_alloc<false>(&tslot, BN);
    tmem_relinquish<false>();
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tacc = tslot;
  const uint32_t idesc = kmajor ? make_idesc_bf16(kBM, BN) & ~((1u << 15) | (1u << 16))
                                : make_idesc_bf16(kBM, BN);
  bool ok = true;
  for (int c = 0; c < nch; c++) {
    const int st = c & 1;
    uint8_t* sa = base + st * L::kStage;
    uint8_t* sb = sa + L::kTileA;
    const int k0 = kbeg + c * kBK;
    // the MMAs that read this stage two chunks ago are done
    if (c >= 2) ok = warp_wait(&bar[st], ((c >> 1) - 1) & 1, &s_abort, err, 11u);
    if constexpr (KS > 0) {
      put(c, sa, sb);
      if (c + 1 < nch) load(c + 1);
    } else {
      for (int idx = tid; idx < (kBM / 8) * kBK; idx += T) {
        const int og = idx & (kBM / 8 - 1), kk = idx / (kBM / 8);
        const int k = k0 + kk;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int m = m0 + og * 8 + i;
          v[i] = (k < kend && m < M) ? op.a(m, k) : 0.0f;
        }
        *reinterpret_cast<uint4*>(sa + tile_off(og >> 3, og & 7, kk, L::kSboA)) = pack8(v);
      }
    }
    if (KS == 0 && op.packed) {
      for (int i = tid; i < (int)(L::kTileB / 16); i += T)
        reinterpret_cast<uint4*>(sb)[i] = __ldg(image(c, i));
    } else if (!kmajor && !op.packed) {
      for (int idx = tid; idx < (BN / 8) * kBK; idx += T) {
        const int og = idx % (BN / 8), kk = idx / (BN / 8);
        const int k = k0 + kk;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int n = n0 + og * 8 + i;
          v[i] = (k < kend && n < N) ? op.b(k, n) : 0.0f;
        }
        *reinterpret_cast<uint4*>(sb + tile_off(og >> 3, og & 7, kk, L::kSboB)) = pack8(v);
      }
    }
    fence_proxy_async();
    if (!__syncthreads_and(ok ? 1 : 0)) {
      ok = false;
      break;
    }
    if (tid == 0) {
      fence_after();
      const uint32_t aa = smem_u32(sa), ba = smem_u32(sb);
#pragma unroll
      for (int t = 0; t < kBK / 16; t++) {
        const uint64_t ad = kmajor ? make_desc(aa + t * 32, 16, 1024)
                                   : make_desc(aa + t * 2 * L::kSboA, 1024, L::kSboA);
        const uint64_t bd = kmajor ? make_desc(ba + t * 32, 16, 1024)
                                   : make_desc(ba + t * 2 * L::kSboB, 1024, L::kSboB);
        mma_f16<false>(tacc, ad, bd, idesc, (c > 0 || t > 0) ? 1u : 0u);
      }
      mma_commit<false>(&bar[st]);
    }
  }
  if (ok && nch > 0) {
    const int c = nch - 1;
    ok = warp_wait(&bar[c & 1], (c >> 1) & 1, &s_abort, err, 12u);
  }
  if (__syncthreads_and(ok ? 1 : 0) && warp < 8) {
    fence_after();
    const int q = warp & 3, h = warp >> 2;
    const int m = m0 + 32 * q + lane;
    // eight columns at a time, the two halves of the warps in turn: all of them
    // have work at 16 columns, and what a column needs is loaded before the
    // stores, which the loads could not pass
    const int cols = min(BN, N - n0);
#pragma unroll 1
    for (int cb = 8 * h; cb < cols; cb += 16) {
      float v[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      if (nch > 0) tmem_ld8(tacc + ((uint32_t)(32 * q) << 16) + (uint32_t)cb, v);
      if (m < M) op.store(op.row(m), n0 + cb, min(8, cols - cb), v, (int)blockIdx.z);
    }
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_dealloc<false>(tacc, BN);
}

// split-K forward: y = act(sum over splits in order + bias)
__global__ void k_conv_fwd_finish(int M, int N, int nsplit, const float* __restrict__ part,
                                  const float* __restrict__ bias, int relu, float* __restrict__ y,
                                  int yC, int yc0, int HW) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= (size_t)M * N) return;
  const int n = (int)(i / M), m = (int)(i - (size_t)n * M);
  float s = 0.0f;
  for (int k = 0; k < nsplit; k++) s += part[((size_t)k * N + n) * M + m];
  s += bias[n];
  if (relu) s = fmaxf(s, 0.0f);
  const int b = m / HW, r = m - b * HW;
  y[(size_t)(b * yC + yc0 + n) * HW + r] = s;
}

// --------------------------------------------------------- plain kernels
// dw = sum over splits (fixed order), db[c] = sum over pixels of dz
__global__ void k_sum_splits(size_t n, int nsplit, const float* __restrict__ part,
                             float* __restrict__ out) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.0f;
  // 16 loads in flight: hundreds of splits of a few hundred weights
  for (int k0 = 0; k0 < nsplit; k0 += 16) {
    float v[16];
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = k0 + k < nsplit ? __ldg(part + (k0 + k) * n + i) : 0.0f;
#pragma unroll
    for (int k = 0; k < 16; k++)
      if (k0 + k < nsplit) s += v[k];
  }
  out[i] = s;
}

// db[c] = sum over pixels of dz, as 256 threads striding over each plane of
// the batch add it: thread t takes pixels t, t + 256, ..., then a butterfly
// within each warp and one over the warps.  A block stands for one of those
// 8 warps (blockIdx.x % 8), so that a channel's sum is not one block's: all its
// threads bring the next 128 steps of the warp's 32 running sums into shared
// memory while the first warp adds the last ones.  16 channels of 256^2,
// batch 8, in one block each: some 600 us; so: 30 us.
constexpr int kBiasSteps = 128;
__global__ void __launch_bounds__(256) k_bias_grad(int B, int HW, View dz, float* __restrict__ part,
                                                   uint32_t* __restrict__ done,
                                                   float* __restrict__ db) {
  __shared__ float stage[2][kBiasSteps][32];
  const int c = blockIdx.x / 8, lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int S = (HW + 255) / 256, total = B * S;  // steps a plane, of the batch
  const int t0 = blockIdx.x % 8 * 32 + lane;       // the thread stood for
  float next[kBiasSteps / 8];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int k = 0; k < kBiasSteps / 8; k++) {
      const int s = s0 + row + 8 * k, b = s / S, i = t0 + 256 * (s - b * S);
      next[k] = s < total && i < HW ? dz.p[(size_t)(b * dz.C + dz.c0 + c) * HW + i] : 0.0f;
    }
  };
  fetch(0);
  float sum = 0.0f;
  int st = 0;
  for (int s0 = 0; s0 < total; s0 += kBiasSteps, st ^= 1) {
#pragma unroll
    for (int k = 0; k < kBiasSteps / 8; k++) stage[st][row + 8 * k][lane] = next[k];
    if (s0 + kBiasSteps < total) fetch(s0 + kBiasSteps);
    __syncthreads();
    if (row == 0) {
#pragma unroll 16
      for (int k = 0; k < kBiasSteps; k++) sum += stage[st][k][lane];
    }
  }
  if (row == 0) {
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) part[blockIdx.x] = sum;
  }
  if (!last_block_done(done, gridDim.x)) return;
  for (int k = threadIdx.x; k < (int)gridDim.x / 8; k += blockDim.x) {
    float w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = __ldcg(part + k * 8 + i);
    db[k] = ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7]));
  }
}

// The resampling kernels: p0 + blockIdx.y = batch and channel (by_planes), a
// thread per pixel of the smaller side.  y = 2x2 average of x (x is H x W, y is
// H/2 x W/2)
__global__ void __launch_bounds__(256) k_pool2(int p0, int C, int H, int W, View x, View y) {
  const int plane = p0 + blockIdx.y, c = plane % C, b = plane / C, Ho = H / 2, Wo = W / 2;
  const float* xp = x.p + (size_t)(b * x.C + x.c0 + c) * H * W;
  float* yp = y.p + (size_t)(b * y.C + y.c0 + c) * Ho * Wo;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Ho * Wo; i += gridDim.x * blockDim.x) {
    const int yo = i / Wo, xo = i - yo * Wo;
    const float2 u = *reinterpret_cast<const float2*>(xp + (size_t)2 * yo * W + 2 * xo);
    const float2 v = *reinterpret_cast<const float2*>(xp + (size_t)(2 * yo + 1) * W + 2 * xo);
    yp[i] = 0.25f * ((u.x + u.y) + (v.x + v.y));
  }
}

// dx += dy / 4 broadcast over each 2x2 block, then masked by the ReLU of act
// (dx's activation)
__global__ void __launch_bounds__(256) k_pool2_bwd(int p0, int C, int H, int W, View dy,
                                                   View dx, View act) {
  const int plane = p0 + blockIdx.y, c = plane % C, b = plane / C, Ho = H / 2, Wo = W / 2;
  const float* gp = dy.p + (size_t)(b * dy.C + dy.c0 + c) * Ho * Wo;
  float* xp = dx.p + (size_t)(b * dx.C + dx.c0 + c) * H * W;
  const float* ap = act.p + (size_t)(b * act.C + act.c0 + c) * H * W;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Ho * Wo; i += gridDim.x * blockDim.x) {
    const int yo = i / Wo, xo = i - yo * Wo;
    const float g = 0.25f * gp[i];
#pragma unroll
    for (int d = 0; d < 2; d++) {
      const size_t o = (size_t)(2 * yo + d) * W + 2 * xo;
      const float2 v = *reinterpret_cast<const float2*>(xp + o);
      const float2 y = *reinterpret_cast<const float2*>(ap + o);
      *reinterpret_cast<float2*>(xp + o) =
          make_float2(y.x > 0.0f ? v.x + g : 0.0f, y.y > 0.0f ? v.y + g : 0.0f);
    }
  }
}

// y = nearest 2x upsample of x (x is H x W)
__global__ void __launch_bounds__(256) k_up2(int p0, int C, int H, int W, View x, View y) {
  const int plane = p0 + blockIdx.y, c = plane % C, b = plane / C, Wo = 2 * W;
  const float* xp = x.p + (size_t)(b * x.C + x.c0 + c) * H * W;
  float* yp = y.p + (size_t)(b * y.C + y.c0 + c) * 4 * H * W;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < H * W; i += gridDim.x * blockDim.x) {
    const int yy = i / W, xx = i - yy * W;
    const float2 v = make_float2(xp[i], xp[i]);
    *reinterpret_cast<float2*>(yp + (size_t)2 * yy * Wo + 2 * xx) = v;
    *reinterpret_cast<float2*>(yp + (size_t)(2 * yy + 1) * Wo + 2 * xx) = v;
  }
}

// dx = sum of dy over each 2x2 block (dx is H x W), masked by the ReLU of act
__global__ void __launch_bounds__(256) k_up2_bwd(int p0, int C, int H, int W, View dy, View dx,
                                                 View act) {
  const int plane = p0 + blockIdx.y, c = plane % C, b = plane / C, Wo = 2 * W;
  const float* gp = dy.p + (size_t)(b * dy.C + dy.c0 + c) * 4 * H * W;
  float* xp = dx.p + (size_t)(b * dx.C + dx.c0 + c) * H * W;
  const float* ap = act.p + (size_t)(b * act.C + act.c0 + c) * H * W;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < H * W; i += gridDim.x * blockDim.x) {
    const int yy = i / W, xx = i - yy * W;
    const float2 u = *reinterpret_cast<const float2*>(gp + (size_t)2 * yy * Wo + 2 * xx);
    const float2 v = *reinterpret_cast<const float2*>(gp + (size_t)(2 * yy + 1) * Wo + 2 * xx);
    xp[i] = ap[i] > 0.0f ? (u.x + u.y) + (v.x + v.y) : 0.0f;
  }
}

// BF16 tile images of the weights as the GEMMs' B operand (forward and data
// gradient), one 16-byte group of eight columns at a time; made when the
// parameters change, so that a tile is a copy instead of 64 strided loads a row.
struct PackEntry {
  size_t w;      // offset of the layer's weights
  int cin, cout, ks, backward;
  int bn, tiles, chunks;
  size_t out;    // offset of the images (16-byte units)
};

__global__ void __launch_bounds__(256) k_pack_weights(const PackEntry* __restrict__ entries,
                                                      const float* __restrict__ params,
                                                      uint4* __restrict__ packed) {
  const PackEntry e = entries[blockIdx.y];
  const int kk = e.ks * e.ks, K = (e.backward ? e.cout : e.cin) * kk;
  const int N = e.backward ? e.cin : e.cout;
  const int per = e.bn / 8 * kBK;  // groups of a tile
  const float* w = params + e.w;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < e.tiles * e.chunks * per;
       i += gridDim.x * blockDim.x) {
    const int tile = i / per, r = i - tile * per;  // n tile * chunks + chunk
    const int og = r % (e.bn / 8), kr = r / (e.bn / 8);
    const int k = (tile % e.chunks) * kBK + kr, n0 = (tile / e.chunks) * e.bn + og * 8;
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int n = n0 + j;
      float x = 0.0f;
      if (k < K && n < N)
        x = e.backward ? w[((size_t)(k / kk) * e.cin + n) * kk + k % kk] : w[(size_t)n * K + k];
      v[j] = x;
    }
    packed[e.out + (size_t)tile * per + tile_off(og >> 3, og & 7, kr, (e.bn / 64) * 1024) / 16] =
        pack8(v);
  }
}

// loss = mean (out - t)^2 (per-block FP64 partials), dout = 2 (out - t) / n
__global__ void k_mse(size_t n, const float* __restrict__ out, const float* __restrict__ t,
                      float* __restrict__ dout, double* __restrict__ part) {
  double s = 0.0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const float d = out[i] - t[i];
    s += (double)d * d;
    if (dout) dout[i] = 2.0f * d / (float)n;
  }
  __shared__ double red[32];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
  }
}

// Adam (Kingma & Ba 2015) with bias correction, FP32 state
__global__ void k_adam(size_t n, float* __restrict__ w, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// ------------------------------------------------------------ host side
struct Ctx {
  cudaStream_t stream;
  uint32_t* err;
  int num_sms;
  float* part;  // split-K scratch for the weight gradient
  size_t part_floats;
  uint32_t* done = nullptr;  // block counter of k_bias_grad
};

inline int tile_columns(int N) { return N <= 64 ? 64 : (N <= 128 ? 128 : 256); }

template <class Op, int BN, int KS>
gv_status launch_gemm_tiled(const Ctx& c, const Op& op, int M, int N, int K, int nsplit) {
  auto kern = k_gemm<Op, BN, KS>;
  const int smem = (int)GemmLayout<BN>::kSmem;
  GV_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int klen = ((K + nsplit - 1) / nsplit + kBK - 1) / kBK * kBK;
  const int nz = (K + klen - 1) / klen;
  dim3 grid((M + kBM - 1) / kBM, (N + BN - 1) / BN, nz);
  kern<<<grid, kGemmThreads, smem, c.stream>>>(op, M, N, K, klen, c.err);
  GV_LAUNCH("k_gemm");
  return GV_OK;
}

template <class Op, int BN>
gv_status launch_gemm_bn(const Ctx& c, const Op& op, int M, int N, int K, int nsplit) {
  if (op.fast && op.ks == 3) return launch_gemm_tiled<Op, BN, 3>(c, op, M, N, K, nsplit);
  if (op.fast && op.ks == 1) return launch_gemm_tiled<Op, BN, 1>(c, op, M, N, K, nsplit);
  return launch_gemm_tiled<Op, BN, 0>(c, op, M, N, K, nsplit);
}

// Column tiles of up to 256, narrower ones where the SMs would not all have a
// CTA: what a chunk costs is its latency and A's staging, hardly its columns
// (the data gradient of the 16^2 level, 16 row tiles of 256 columns and 36
// chunks: 101 us in 16 CTAs, 53 in 64).
template <class Op>
gv_status launch_gemm(const Ctx& c, const Op& op, int M, int N, int K, int nsplit = 1) {
  int bn = tile_columns(N);
  while (bn > 64 && ((M + kBM - 1) / kBM) * ((N + bn - 1) / bn) * nsplit < c.num_sms) bn /= 2;
  if (bn == 64) return launch_gemm_bn<Op, 64>(c, op, M, N, K, nsplit);
  if (bn == 128) return launch_gemm_bn<Op, 128>(c, op, M, N, K, nsplit);
  return launch_gemm_bn<Op, 256>(c, op, M, N, K, nsplit);
}

// launch(grid, first plane) of a resampling kernel: n pixels a plane, as many
// planes at once as a grid's second dimension takes
template <class F>
gv_status by_planes(const char* name, int n, int planes, F&& launch) {
  constexpr int kMost = 65535;
  for (int p0 = 0; p0 < planes; p0 += kMost) {
    launch(dim3((unsigned)std::min((n + 255) / 256, 64), (unsigned)std::min(planes - p0, kMost)),
           p0);
    GV_LAUNCH(name);
  }
  return GV_OK;
}

inline int ew_blocks(size_t n, const Ctx& c) {
  return (int)std::max<size_t>(1, std::min<size_t>((n + 255) / 256, (size_t)8 * c.num_sms));
}

gv_status conv_forward(const Ctx& c, View x, const float* w, const uint4* packed,
                       const float* bias, View y, int B, int Cin, int Cout, int H, int W, int ks,
                       int relu) {
  const int M = B * H * W, N = Cout, K = Cin * ks * ks;
  // a grid of fewer tiles than SMs (deep levels, small batches) splits K
  // over up to two CTAs per SM, at least two K blocks a split
  const int bn = tile_columns(N);
  const int tiles = ((M + kBM - 1) / kBM) * ((N + bn - 1) / bn);
  int nsplit = 1;
  if (c.part && tiles < c.num_sms) {
    nsplit = std::min(K / (2 * kBK), (2 * c.num_sms + tiles - 1) / tiles);
    nsplit = std::max(1, std::min<int>(nsplit, (int)(c.part_floats / ((size_t)M * N))));
  }
  ConvFwdOp op{x.p, x.C, x.c0, w, packed, bias, y.p, y.C, y.c0, Cin, Cout, H, W, ks, relu,
               nsplit > 1 ? c.part : nullptr, M, rows_of_eight(x.p, W)};
  gv_status s = launch_gemm(c, op, M, N, K, nsplit);
  if (s != GV_OK || nsplit <= 1) return s;
  // the kernel launched ceil(K / klen) splits; sum exactly those
  const int klen = ((K + nsplit - 1) / nsplit + kBK - 1) / kBK * kBK;
  const int nz = (K + klen - 1) / klen;
  k_conv_fwd_finish<<<(unsigned)(((size_t)M * N + 255) / 256), 256, 0, c.stream>>>(
      M, N, nz, c.part, bias, relu, y.p, y.C, y.c0, H * W);
  GV_LAUNCH("k_conv_fwd_finish");
  return GV_OK;
}

gv_status conv_backward_data(const Ctx& c, View dz, const float* w, const uint4* packed, View dx,
                             View act, int B, int Cin, int Cout, int H, int W, int ks) {
  ConvBwdDataOp op{dz.p, dz.C, dz.c0, w, packed, dx.p, dx.C, dx.c0, act.p, act.C, act.c0, Cin, Cout,
                   H, W, ks, rows_of_eight(dz.p, W)};
  return launch_gemm(c, op, B * H * W, Cin, Cout * ks * ks);
}

// FP32 scratch of a weight gradient: a whole split's partial sums, or the bias
// gradient's 8 a channel
inline size_t weight_scratch(int Cin, int Cout, int ks) {
  return (size_t)Cout * std::max<size_t>((size_t)Cin * ks * ks, 8);
}

gv_status conv_backward_weight(const Ctx& c, View x, View dz, float* dw, float* db, int B,
                               int Cin, int Cout, int H, int W, int ks) {
  const int M = Cin * ks * ks, N = Cout, K = B * H * W;
  const int tiles = ((M + kBM - 1) / kBM) * ((N + 255) / 256);
  const size_t wn = (size_t)M * N;
  int nsplit = std::max(1, std::min(K / 1024, (2 * c.num_sms + tiles - 1) / tiles));
  nsplit = std::max(1, std::min<int>(nsplit, (int)(c.part_floats / wn)));
  ConvBwdWeightOp op{x.p, x.C, x.c0, dz.p, dz.C, dz.c0, c.part, Cin, Cout, H, W, ks,
                     rows_of_eight(x.p, W) && rows_of_eight(dz.p, W)};
  gv_status s = launch_gemm(c, op, M, N, K, nsplit);
  if (s != GV_OK) return s;
  // the kernel launched ceil(K / klen) splits; sum exactly those
  const int klen = ((K + nsplit - 1) / nsplit + kBK - 1) / kBK * kBK;
  const int nz = (K + klen - 1) / klen;
  k_sum_splits<<<(unsigned)((wn + 255) / 256), 256, 0, c.stream>>>(wn, nz, c.part, dw);
  GV_LAUNCH("k_sum_splits");
  // the splits' scratch is free again
  k_bias_grad<<<8 * Cout, 256, 0, c.stream>>>(B, H * W, dz, c.part, c.done, db);
  GV_LAUNCH("k_bias_grad");
  return GV_OK;
}

// ----------------------------------------------------------------- U-Net
struct Layer {
  int cin, cout, ks, relu, side;
  size_t w, b;  // offsets into the parameter vector
};

struct UNet {
  int H = 0, W = 0, cin = 0, c0 = 0, L = 0, maxB = 0;
  std::vector<Layer> layers;
  size_t nparams = 0;
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  int step = 0;
  // activations and gradients (device), see the layout comment at the top
  std::vector<float*> in, a, enc, cat, b, dec;      // per level
  std::vector<float*> din, da, denc, dcat, dbuf, ddec;
  float *out = nullptr, *dout = nullptr;
  double* loss_part = nullptr;
  double* h_loss = nullptr;
  uint32_t* err = nullptr;
  float* part = nullptr;
  size_t part_floats = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 0;
  std::vector<void*> allocs;
  // forward passes captured as CUDA graphs, one per batch size (the pass
  // only reads and writes the network's own buffers, so a graph stays valid)
  std::vector<cudaGraphExec_t> fwd_exec;
  std::vector<int64_t> fwd_launches;
  cudaStream_t cap = nullptr;
  // the weight gradients' stream, beside the chain of the data gradients
  cudaStream_t side = nullptr;
  cudaEvent_t ready = nullptr;

  int C(int l) const { return c0 << l; }
  int S(int l) const { return H >> l; }
  // BF16 tile images of the weights: forward, then data gradient, per layer
  std::vector<PackEntry> entries;
  PackEntry* d_entries = nullptr;
  uint4* packed = nullptr;
  Ctx ctx() const { return Ctx{stream, err, num_sms, part, part_floats, err + 1}; }
  const uint4* image(int layer, int backward) const {
    return packed + entries[2 * layer + backward].out;
  }
  // after every change of the parameters
  gv_status pack() {
    k_pack_weights<<<dim3(32, (unsigned)entries.size()), 256, 0, stream>>>(d_entries, params,
                                                                           packed);
    GV_LAUNCH("k_pack_weights");
    return GV_OK;
  }

  gv_status alloc(float** p, size_t n) {
    GV_CUDA(cudaMalloc(p, std::max<size_t>(n, 1) * sizeof(float)));
    GV_CUDA(cudaMemsetAsync(*p, 0, std::max<size_t>(n, 1) * sizeof(float), stream));
    allocs.push_back(*p);
    return GV_OK;
  }
  ~UNet() {
    for (cudaGraphExec_t g : fwd_exec)
      if (g) cudaGraphExecDestroy(g);
    if (cap) cudaStreamDestroy(cap);
    if (side) cudaStreamDestroy(side);
    if (ready) cudaEventDestroy(ready);
    for (void* p : allocs) cudaFree(p);
    if (h_loss) cudaFreeHost(h_loss);
  }

  // layer index helpers: enc l -> 2l, 2l+1; dec l (l = L-2..0) -> 2L + 2(L-2-l), +1; out last
  int enc_layer(int l, int j) const { return 2 * l + j; }
  int dec_layer(int l, int j) const { return 2 * L + 2 * (L - 2 - l) + j; }
  int out_layer() const { return 2 * L + 2 * (L - 1); }

  gv_status build(const gv_unet_desc& d) {
    H = d.height;
    W = d.width;
    cin = d.in_channels;
    c0 = d.base_channels;
    L = d.levels;
    maxB = d.max_batch;
    size_t off = 0;
    auto add = [&](int ci, int co, int ks, int relu, int side) {
      Layer ly{ci, co, ks, relu, side, off, off + (size_t)co * ci * ks * ks};
      off = ly.b + co;
      layers.push_back(ly);
    };
    for (int l = 0; l < L; l++) {
      add(l == 0 ? cin : C(l - 1), C(l), 3, 1, S(l));
      add(C(l), C(l), 3, 1, S(l));
    }
    for (int l = L - 2; l >= 0; l--) {
      add(C(l + 1) + C(l), C(l), 3, 1, S(l));
      add(C(l), C(l), 3, 1, S(l));
    }
    add(C(0), 1, 1, 0, S(0));
    nparams = off;
    GV_TRY(alloc(&params, nparams));
    GV_TRY(alloc(&grads, nparams));
    GV_TRY(alloc(&m, nparams));
    GV_TRY(alloc(&v, nparams));
    // He-normal weights, zero biases (seeded)
    std::vector<float> h(nparams, 0.0f);
    std::mt19937_64 rng(d.seed);
    for (const Layer& ly : layers) {
      std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)(ly.cin * ly.ks * ly.ks)));
      for (size_t i = ly.w; i < ly.b; i++) h[i] = nd(rng);
    }
    GV_CUDA(cudaMemcpyAsync(params, h.data(), nparams * sizeof(float), cudaMemcpyHostToDevice,
                            stream));
    const size_t B = maxB;
    in.resize(L);
    a.resize(L);
    enc.resize(L);
    cat.resize(L);
    b.resize(L);
    dec.resize(L);
    din.resize(L);
    da.resize(L);
    denc.resize(L);
    dcat.resize(L);
    dbuf.resize(L);
    ddec.resize(L);
    for (int l = 0; l < L; l++) {
      const size_t px = B * (size_t)S(l) * S(l);
      const int cin_l = l == 0 ? cin : C(l - 1);
      GV_TRY(alloc(&in[l], px * cin_l));
      GV_TRY(alloc(&a[l], px * C(l)));
      GV_TRY(alloc(&din[l], px * cin_l));
      GV_TRY(alloc(&da[l], px * C(l)));
      if (l < L - 1) {
        // enc_l lives in channels [C(l+1), C(l+1) + C(l)) of the concat buffer
        GV_TRY(alloc(&cat[l], px * (C(l + 1) + C(l))));
        GV_TRY(alloc(&dcat[l], px * (C(l + 1) + C(l))));
        GV_TRY(alloc(&b[l], px * C(l)));
        GV_TRY(alloc(&dbuf[l], px * C(l)));
        GV_TRY(alloc(&dec[l], px * C(l)));
        GV_TRY(alloc(&ddec[l], px * C(l)));
      } else {
        GV_TRY(alloc(&enc[l], px * C(l)));
        GV_TRY(alloc(&denc[l], px * C(l)));
      }
    }
    GV_TRY(alloc(&out, B * (size_t)H * W));
    GV_TRY(alloc(&dout, B * (size_t)H * W));
    part_floats = (size_t)4 << 20;  // 16 MB of split-K partials
    for (const Layer& ly : layers)
      part_floats = std::max(part_floats, weight_scratch(ly.cin, ly.cout, ly.ks));
    GV_TRY(alloc(&part, part_floats));
    GV_CUDA(cudaMalloc(&loss_part, sizeof(double) * 1024));
    allocs.push_back(loss_part);
    GV_CUDA(cudaMalloc(&err, 2 * sizeof(uint32_t)));  // error word, block counter
    allocs.push_back(err);
    GV_CUDA(cudaMemsetAsync(err, 0, 2 * sizeof(uint32_t), stream));
    size_t images = 0;
    for (const Layer& ly : layers)
      for (int back = 0; back < 2; back++) {
        const int N = back ? ly.cin : ly.cout, K = (back ? ly.cout : ly.cin) * ly.ks * ly.ks;
        // whole tiles of whatever width the launch takes
        const int bn = 64, chunks = (K + kBK - 1) / kBK;
        const int tiles = (N + tile_columns(N) - 1) / tile_columns(N) * (tile_columns(N) / bn);
        entries.push_back({ly.w, ly.cin, ly.cout, ly.ks, back, bn, tiles, chunks, images});
        images += (size_t)tiles * chunks * (bn / 8) * kBK;
      }
    GV_CUDA(cudaMalloc(&packed, sizeof(uint4) * images));
    allocs.push_back(packed);
    GV_CUDA(cudaMalloc(&d_entries, sizeof(PackEntry) * entries.size()));
    allocs.push_back(d_entries);
    GV_CUDA(cudaMemcpy(d_entries, entries.data(), sizeof(PackEntry) * entries.size(),
                       cudaMemcpyHostToDevice));
    GV_TRY(pack());
    GV_CUDA(cudaMallocHost(&h_loss, sizeof(double) * 1024));
    return GV_OK;
  }

  // views of enc_l (inside the concat buffer for l < L-1) and its gradient
  View enc_view(int l) const {
    if (l < L - 1) return View{cat[l], C(l + 1) + C(l), C(l + 1)};
    return View{enc[l], C(l), 0};
  }
  View denc_view(int l) const {
    if (l < L - 1) return View{dcat[l], C(l + 1) + C(l), C(l + 1)};
    return View{denc[l], C(l), 0};
  }
  View dec_view(int l) const { return l == L - 1 ? enc_view(l) : View{dec[l], C(l), 0}; }
  View ddec_view(int l) const { return l == L - 1 ? denc_view(l) : View{ddec[l], C(l), 0}; }

  // The input is copied into the network's buffer, then the pass is one
  // graph launch (captured on first use for this batch size on a private
  // stream; a batch-1 pass is some 40 small kernels whose launch latency
  // would otherwise set its time).
  gv_status forward(const float* d_in, int B) {
    GV_CUDA(cudaMemcpyAsync(in[0], d_in, sizeof(float) * B * cin * H * W,
                            cudaMemcpyDeviceToDevice, stream));
    if (fwd_exec.empty()) {
      fwd_exec.assign(maxB + 1, nullptr);
      fwd_launches.assign(maxB + 1, 0);
    }
    if (!fwd_exec[B]) {
      if (!cap) GV_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
      const cudaStream_t saved = stream;
      const int64_t l0 = gv_launch_count();
      stream = cap;
      cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeRelaxed);
      if (e != cudaSuccess) {
        stream = saved;
        return cuda_fail(e, "cudaStreamBeginCapture (U-Net forward)");
      }
      const gv_status s = forward_pass(B);
      cudaGraph_t g = nullptr;
      e = cudaStreamEndCapture(cap, &g);
      stream = saved;
      const int64_t nl = gv_launch_count() - l0;
      add_launches(-nl);  // counted again at each replay
      if (s != GV_OK) {
        if (g) cudaGraphDestroy(g);
        return s;
      }
      if (e != cudaSuccess) return cuda_fail(e, "cudaStreamEndCapture (U-Net forward)");
      cudaGraphExec_t x = nullptr;
      e = cudaGraphInstantiate(&x, g, 0);
      cudaGraphDestroy(g);
      if (e != cudaSuccess) return cuda_fail(e, "cudaGraphInstantiate (U-Net forward)");
      fwd_exec[B] = x;
      fwd_launches[B] = nl;
    }
    GV_CUDA(cudaGraphLaunch(fwd_exec[B], stream));
    add_launches(fwd_launches[B]);
    return GV_OK;
  }

  gv_status layer_forward(const Ctx& c, int k, View x, View y, int B, int s) {
    const Layer& ly = layers[k];
    return conv_forward(c, x, params + ly.w, image(k, 0), params + ly.b, y, B, ly.cin, ly.cout, s,
                        s, ly.ks, ly.relu);
  }

  // the forward pass on the network's input buffer in[0]
  gv_status forward_pass(int B) {
    const Ctx c = ctx();
    for (int l = 0; l < L; l++) {
      const int s = S(l), ci = l == 0 ? cin : C(l - 1);
      GV_TRY(layer_forward(c, enc_layer(l, 0), View{in[l], ci, 0}, View{a[l], C(l), 0}, B, s));
      GV_TRY(layer_forward(c, enc_layer(l, 1), View{a[l], C(l), 0}, enc_view(l), B, s));
      if (l + 1 < L) {
        GV_TRY(by_planes("k_pool2", s * s / 4, B * C(l), [&](dim3 grid, int p0) {
          k_pool2<<<grid, 256, 0, stream>>>(p0, C(l), s, s, enc_view(l), View{in[l + 1], C(l), 0});
        }));
      }
    }
    for (int l = L - 2; l >= 0; l--) {
      const int s = S(l), cc = C(l + 1) + C(l);
      GV_TRY(by_planes("k_up2", s * s / 4, B * C(l + 1), [&](dim3 grid, int p0) {
        k_up2<<<grid, 256, 0, stream>>>(p0, C(l + 1), s / 2, s / 2, dec_view(l + 1),
                                        View{cat[l], cc, 0});
      }));
      GV_TRY(layer_forward(c, dec_layer(l, 0), View{cat[l], cc, 0}, View{b[l], C(l), 0}, B, s));
      GV_TRY(layer_forward(c, dec_layer(l, 1), View{b[l], C(l), 0}, dec_view(l), B, s));
    }
    return layer_forward(c, out_layer(), dec_view(0), View{out, 1, 0}, B, H);
  }

  // weight, bias and data gradient of layer k from dz (its pre-activation's
  // gradient); dx is masked by the ReLU of act where act is set
  // The weight gradients go to the side stream: nothing of the chain waits for
  // them, no buffer that they read (activations, gradients) is written again
  // before the join, and they alone use the splits' scratch meanwhile.  Deep
  // levels have 16 to 72 CTAs a GEMM, so that the two together fill the chip
  // (a training step of the 256^2 network, batch 8:
  // 2670 us one after the other, 2480 so).
  gv_status layer_backward(const Ctx& c, int k, View x, View dz, View dx, View act, int B, int s) {
    const Layer& ly = layers[k];
    GV_CUDA(cudaEventRecord(ready, stream));  // dz is there
    GV_CUDA(cudaStreamWaitEvent(side, ready, 0));
    Ctx cw = c;
    cw.stream = side;
    GV_TRY(conv_backward_weight(cw, x, dz, grads + ly.w, grads + ly.b, B, ly.cin, ly.cout, s, s,
                                ly.ks));
    if (!dx.p) return GV_OK;
    return conv_backward_data(c, dz, params + ly.w, image(k, 1), dx, act, B, ly.cin, ly.cout, s, s,
                              ly.ks);
  }

  // gradients of the loss with respect to every parameter, given dout.  Every
  // gradient of an activation is masked by that activation's ReLU where it is
  // made (the data-gradient GEMM's epilogue or the resampling), so it is the
  // next layer's dz as it stands.
  gv_status backward(int B) {
    if (!side) GV_CUDA(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    if (!ready) GV_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    const gv_status s = backward_pass(B);
    // joined on every way out
    GV_CUDA(cudaEventRecord(ready, side));
    GV_CUDA(cudaStreamWaitEvent(stream, ready, 0));
    return s;
  }

  gv_status backward_pass(int B) {
    const Ctx c = ctx();
    const View none{nullptr, 0, 0};
    GV_TRY(layer_backward(c, out_layer(), dec_view(0), View{dout, 1, 0}, ddec_view(0), dec_view(0),
                          B, H));
    for (int l = 0; l <= L - 2; l++) {
      const int s = S(l), cc = C(l + 1) + C(l);
      const View bv{b[l], C(l), 0}, dbv{dbuf[l], C(l), 0}, dcatv{dcat[l], cc, 0};
      GV_TRY(layer_backward(c, dec_layer(l, 1), bv, ddec_view(l), dbv, bv, B, s));
      GV_TRY(layer_backward(c, dec_layer(l, 0), View{cat[l], cc, 0}, dbv, dcatv, none, B, s));
      // the upsampled part of the concat feeds dec_{l+1}
      GV_TRY(by_planes("k_up2_bwd", s * s / 4, B * C(l + 1), [&](dim3 grid, int p0) {
        k_up2_bwd<<<grid, 256, 0, stream>>>(p0, C(l + 1), s / 2, s / 2, dcatv, ddec_view(l + 1),
                                            dec_view(l + 1));
      }));
    }
    for (int l = L - 1; l >= 0; l--) {
      const int s = S(l), ci = l == 0 ? cin : C(l - 1);
      if (l + 1 < L) {
        // enc_l also feeds the pool of level l+1: add that gradient
        GV_TRY(by_planes("k_pool2_bwd", s * s / 4, B * C(l), [&](dim3 grid, int p0) {
          k_pool2_bwd<<<grid, 256, 0, stream>>>(p0, C(l), s, s, View{din[l + 1], C(l), 0},
                                                denc_view(l), enc_view(l));
        }));
      }
      const View av{a[l], C(l), 0}, dav{da[l], C(l), 0};
      GV_TRY(layer_backward(c, enc_layer(l, 1), av, denc_view(l), dav, av, B, s));
      GV_TRY(layer_backward(c, enc_layer(l, 0), View{in[l], ci, 0}, dav,
                            l > 0 ? View{din[l], ci, 0} : none, none, B, s));
    }
    return GV_OK;
  }

  // the loss' partial sums on their way to the host (loss_value, after a
  // synchronisation) and its gradient in dout
  static constexpr int kLossBlocks = 256;
  gv_status loss_launch(const float* d_target, int B) {
    const size_t n = (size_t)B * H * W;
    k_mse<<<kLossBlocks, 256, 0, stream>>>(n, out, d_target, dout, loss_part);
    GV_LAUNCH("k_mse");
    GV_CUDA(cudaMemcpyAsync(h_loss, loss_part, sizeof(double) * kLossBlocks,
                            cudaMemcpyDeviceToHost, stream));
    return GV_OK;
  }
  double loss_value(int B) const {
    double s = 0.0;
    for (int i = 0; i < kLossBlocks; i++) s += h_loss[i];
    return s / (double)((size_t)B * H * W);
  }

  gv_status adam(float lr) {
    step++;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.0f - std::pow(b1, (float)step), c2 = 1.0f - std::pow(b2, (float)step);
    const Ctx c = ctx();
    k_adam<<<ew_blocks(nparams, c), 256, 0, stream>>>(nparams, params, grads, m, v, lr, b1, b2,
                                                      eps, c1, c2);
    GV_LAUNCH("k_adam");
    return pack();
  }

  gv_status check() {
    uint32_t e = 0;
    GV_CUDA(cudaMemcpyAsync(&e, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream));
    GV_CUDA(cudaStreamSynchronize(stream));
    if (e) {
      GV_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), stream));
      set_error("a tensor-core GEMM gave up on a bounded wait (device error word " +
                std::to_string(e) + ")");
      return GV_ERR_DEVICE;
    }
    return GV_OK;
  }
};

}  // namespace cnn
}  // namespace gv

struct gv_unet {
  gv::cnn::UNet net;
};

namespace {

gv_status check_batch(const gv_unet* n, int32_t batch) {
  if (!n || batch < 1 || batch > n->net.maxB) {
    gv::set_error("null network or batch outside [1, max_batch]");
    return GV_ERR_INVALID;
  }
  return GV_OK;
}

gv::cnn::Ctx standalone_ctx(void* stream, uint32_t* err, float* part, size_t part_floats) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return gv::cnn::Ctx{(cudaStream_t)stream, err, sms, part, part_floats, err + 1};
}

}  // namespace

extern "C" {

gv_status gv_unet_create(const gv_unet_desc* d, gv_unet** out) {
  if (!d || !out) {
    gv::set_error("null descriptor or output");
    return GV_ERR_INVALID;
  }
  *out = nullptr;
  if (d->levels < 1 || d->levels > 6 || d->base_channels < 8 || d->base_channels % 8 != 0 ||
      d->in_channels < 1 || d->max_batch < 1 || d->height != d->width ||
      (d->height >> (d->levels - 1)) < 2 || (d->height % (1 << (d->levels - 1))) != 0 ||
      (d->base_channels << (d->levels - 1)) > 256) {
    gv::set_error("unsupported network shape (square image divisible by 2^(levels-1), "
                  "base channels a multiple of 8, at most 256 channels)");
    return GV_ERR_INVALID;
  }
  gv_unet* n = new gv_unet();
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n->net.num_sms, cudaDevAttrMultiProcessorCount, dev);
  gv_status s = n->net.build(*d);
  if (s == GV_OK) {
    cudaError_t e = cudaStreamSynchronize(n->net.stream);
    if (e != cudaSuccess) s = gv::cuda_fail(e, "unet set-up");
  }
  if (s != GV_OK) {
    delete n;
    return s;
  }
  *out = n;
  return GV_OK;
}

gv_status gv_unet_destroy(gv_unet* n) {
  if (!n) return GV_OK;
  cudaStreamSynchronize(n->net.stream);
  delete n;
  return GV_OK;
}

gv_status gv_unet_set_stream(gv_unet* n, void* stream) {
  if (!n) return GV_ERR_INVALID;
  n->net.stream = (cudaStream_t)stream;
  return GV_OK;
}

gv_status gv_unet_num_params(const gv_unet* n, int64_t* count) {
  if (!n || !count) return GV_ERR_INVALID;
  *count = (int64_t)n->net.nparams;
  return GV_OK;
}

gv_status gv_unet_get_params(gv_unet* n, float* d_out) {
  if (!n || !d_out) return GV_ERR_INVALID;
  GV_CUDA(cudaMemcpyAsync(d_out, n->net.params, sizeof(float) * n->net.nparams,
                          cudaMemcpyDeviceToDevice, n->net.stream));
  GV_CUDA(cudaStreamSynchronize(n->net.stream));
  return GV_OK;
}

gv_status gv_unet_set_params(gv_unet* n, const float* d_in) {
  if (!n || !d_in) return GV_ERR_INVALID;
  GV_CUDA(cudaMemcpyAsync(n->net.params, d_in, sizeof(float) * n->net.nparams,
                          cudaMemcpyDeviceToDevice, n->net.stream));
  GV_CUDA(cudaMemsetAsync(n->net.m, 0, sizeof(float) * n->net.nparams, n->net.stream));
  GV_CUDA(cudaMemsetAsync(n->net.v, 0, sizeof(float) * n->net.nparams, n->net.stream));
  n->net.step = 0;
  GV_TRY(n->net.pack());
  GV_CUDA(cudaStreamSynchronize(n->net.stream));
  return GV_OK;
}

gv_status gv_unet_get_grads(gv_unet* n, float* d_out) {
  if (!n || !d_out) return GV_ERR_INVALID;
  GV_CUDA(cudaMemcpyAsync(d_out, n->net.grads, sizeof(float) * n->net.nparams,
                          cudaMemcpyDeviceToDevice, n->net.stream));
  GV_CUDA(cudaStreamSynchronize(n->net.stream));
  return GV_OK;
}

gv_status gv_unet_forward(gv_unet* n, const float* d_in, int32_t batch, float* d_out) {
  GV_TRY(check_batch(n, batch));
  if (!d_in || !d_out) return GV_ERR_INVALID;
  GV_TRY(n->net.forward(d_in, batch));
  GV_CUDA(cudaMemcpyAsync(d_out, n->net.out, sizeof(float) * batch * n->net.H * n->net.W,
                          cudaMemcpyDeviceToDevice, n->net.stream));
  return n->net.check();
}

gv_status gv_unet_loss_grad(gv_unet* n, const float* d_in, const float* d_target, int32_t batch,
                            double* loss) {
  GV_TRY(check_batch(n, batch));
  if (!d_in || !d_target) return GV_ERR_INVALID;
  GV_TRY(n->net.forward(d_in, batch));
  GV_TRY(n->net.loss_launch(d_target, batch));
  GV_TRY(n->net.backward(batch));
  GV_TRY(n->net.check());
  if (loss) *loss = n->net.loss_value(batch);
  return GV_OK;
}

gv_status gv_unet_train_step(gv_unet* n, const float* d_in, const float* d_target, int32_t batch,
                             float lr, double* loss) {
  GV_TRY(check_batch(n, batch));
  if (!d_in || !d_target) return GV_ERR_INVALID;
  GV_TRY(n->net.forward(d_in, batch));
  GV_TRY(n->net.loss_launch(d_target, batch));
  GV_TRY(n->net.backward(batch));
  GV_TRY(n->net.adam(lr));
  GV_TRY(n->net.check());
  if (loss) *loss = n->net.loss_value(batch);
  return GV_OK;
}

gv_status gv_conv2d_forward(const float* x, const float* w, const float* bias, float* y,
                            int32_t B, int32_t Cin, int32_t Cout, int32_t H, int32_t W,
                            int32_t ks, int32_t relu, void* stream) {
  if (!x || !w || !bias || !y || B < 1 || Cin < 1 || Cout < 1 || H < 1 || W < 1 ||
      (ks != 1 && ks != 3)) {
    gv::set_error("invalid convolution arguments");
    return GV_ERR_INVALID;
  }
  uint32_t* err = nullptr;
  GV_CUDA(cudaMalloc(&err, 2 * sizeof(uint32_t)));
  GV_CUDA(cudaMemsetAsync(err, 0, 2 * sizeof(uint32_t), (cudaStream_t)stream));
  const gv::cnn::Ctx c = standalone_ctx(stream, err, nullptr, 0);
  gv_status s = gv::cnn::conv_forward(c, gv::cnn::View{(float*)x, Cin, 0}, w, nullptr, bias,
                                      gv::cnn::View{y, Cout, 0}, B, Cin, Cout, H, W, ks, relu);
  uint32_t e = 0;
  cudaMemcpyAsync(&e, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  cudaStreamSynchronize((cudaStream_t)stream);
  cudaFree(err);
  if (s == GV_OK && e) {
    gv::set_error("convolution gave up on a bounded wait");
    s = GV_ERR_DEVICE;
  }
  return s;
}

gv_status gv_conv2d_backward(const float* x, const float* w, const float* dz, float* dx,
                             float* dw, float* db, int32_t B, int32_t Cin, int32_t Cout,
                             int32_t H, int32_t W, int32_t ks, void* stream) {
  if (!x || !w || !dz || !dx || !dw || !db || B < 1 || Cin < 1 || Cout < 1 || H < 1 || W < 1 ||
      (ks != 1 && ks != 3)) {
    gv::set_error("invalid convolution arguments");
    return GV_ERR_INVALID;
  }
  uint32_t* err = nullptr;
  float* part = nullptr;
  const size_t part_floats =
      std::max((size_t)4 << 20, gv::cnn::weight_scratch(Cin, Cout, ks));
  GV_CUDA(cudaMalloc(&err, 2 * sizeof(uint32_t)));
  GV_CUDA(cudaMalloc(&part, sizeof(float) * part_floats));
  GV_CUDA(cudaMemsetAsync(err, 0, 2 * sizeof(uint32_t), (cudaStream_t)stream));
  const gv::cnn::Ctx c = standalone_ctx(stream, err, part, part_floats);
  gv_status s = gv::cnn::conv_backward_data(c, gv::cnn::View{(float*)dz, Cout, 0}, w, nullptr,
                                            gv::cnn::View{dx, Cin, 0},
                                            gv::cnn::View{nullptr, 0, 0}, B, Cin, Cout, H, W, ks);
  if (s == GV_OK)
    s = gv::cnn::conv_backward_weight(c, gv::cnn::View{(float*)x, Cin, 0},
                                      gv::cnn::View{(float*)dz, Cout, 0}, dw, db, B, Cin, Cout, H,
                                      W, ks);
  uint32_t e = 0;
  cudaMemcpyAsync(&e, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  cudaStreamSynchronize((cudaStream_t)stream);
  cudaFree(err);
  cudaFree(part);
  if (s == GV_OK && e) {
    gv::set_error("convolution gave up on a bounded wait");
    s = GV_ERR_DEVICE;
  }
  return s;
}

}  // extern "C"
