// DChi2 (src/functions.cu:3698-3791) as a non-uniform FFT: the same sum over
// visibilities for every pixel,
//   S(i,j) = sum_k Re(conj(c_k) e^{2 pi i (x_j u_k + y_i v_k + (z - 1) w_k)}),
// with the work of one local spreading per visibility and two pruned FFTs per
// channel instead of one product per pixel and visibility.
//
//  1. k_nu_spread  every visibility is spread over 8 x 8 cells of a grid of
//                  twice the image's sides with the kernel
//                  e^{beta (sqrt(1 - t^2) - 1)} (Barnett, Magland and af
//                  Klinteberg, "A parallel non-uniform fast Fourier transform
//                  library based on an exponential of semicircle kernel",
//                  SIAM J. Sci. Comput. 41, 2019);
//  2. k_nu_merge   the tiles' sums are added into the rows and columns of the
//                  grid that the data cover;
//  3. k_nu_rows    row FFTs of the covered rows, the image's N of 2N outputs;
//  4. k_nu_cols    column FFTs, the kernel's correction, the w-term, beam,
//                  mask and chain rule, summed over the channels.
//
// The w-term is a Chebyshev series (the Jacobi-Anger expansion): with
// s = w / wmax in [-1, 1] and a = 2 pi wmax (z - 1) per pixel,
//   e^{i a s} = sum_n (2 - [n = 0]) i^n J_n(a) T_n(s).
// Only Re is needed, so the even terms need the real part of their plane's
// transform and the odd ones the imaginary part: one complex FFT carries an
// even and an odd term, the grid being the Hermitian part of the one plus the
// anti-Hermitian part of the other.  2 kPairs terms leave
// 2 (A/2)^(2 kPairs) / (2 kPairs)!, A = max |a|; problems whose A needs more
// than 4 pairs keep the direct sums.
//
// All arithmetic is FP32 on exact 32-bit fixed-point grid positions; every
// sum is taken in a fixed order (no atomics), so results repeat bit for bit.
// Against 64-bit sums the gradient is 1.1 to 1.7e-7 off in the 2-norm (256^2
// and 1024^2), where the tensor-core sum is 1.2 to 1.4e-6 off.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft.cuh"
#include "gv_internal.cuh"

namespace gv {

// Work of one warp of k_nu_spread: `count` consecutive visibilities, all
// with their first cell in one 8 x 8 tile of the doubled grid.
struct NuTask {
  uint32_t begin;
  int count;
};

struct NuPlan {
  int pairs = 0;           // complex FFTs per channel
  float wmax = 0.0f;
  int cmin = 0, ncol = 0;  // covered columns (signed), ncol even
  int rmin = 0, nrow = 0;  // covered rows (signed)
  int wrap = 0;            // cells beyond +-N: the grid's period matters
  int tx0 = 0, ntx = 0, ty0 = 0, nty = 0;  // tiles in use
  std::vector<int> task_off;   // [C + 1]
  std::vector<int> groups;     // channel group boundaries
  NuTask* d_tasks = nullptr;
  int* d_slot_off = nullptr;   // [C nty ntx + 1] tasks of each tile
  float2* d_slots = nullptr;   // per task: [pair][plane][225] sums
  float2* d_F = nullptr;       // [channel of the group][pair][nrow][ncol]
  float2* d_H = nullptr;       // [channel of the group][pair][nrow][N]
  float2* d_turn = nullptr;    // [N] e^{2 pi i (j - N/2) / 2N}
  float* d_corr = nullptr;     // [N] 1 / kernel transform
  float2* d_coef = nullptr;    // [pair][MN] w-term coefficients (k_nu_coefficients)
  float* d_fac = nullptr;      // [channel of the group][MN] k_nu_factors
  float coef[4][12];           // the taps' polynomials (tap_polynomials)
};

namespace {

constexpr int kTaps = 8;
constexpr int kTileSide = 15;  // 8 first cells + 7
constexpr int kTilePts = kTileSide * kTileSide;
constexpr int kSpreadWarps = 4;
constexpr int kMaxPairs = 4;
constexpr double kBeta = 2.30 * kTaps;
constexpr int kPolyHalf = 6;  // even and odd coefficients of a tap's polynomial
// truncation of the w series (of the largest term, at the image's corner)
constexpr double kWTol = 3e-7;
// bound of the slots + grids of one channel group
constexpr size_t kWorkspace = size_t(4) << 30;

struct SpreadArgs {
  const uint4* __restrict__ ph;
  const float2* __restrict__ cvr;
  const float4* __restrict__ deg;
  const float2* __restrict__ vo;
  const NuTask* __restrict__ tasks;
  int ntasks;
  float2* __restrict__ slots;
  int mode;        // of the DChi2 engines: 0/1 residuals, 2 Vo, 3 weights, 4 conjugated residuals
  int sh;          // fraction bits of a fixed-point position on the doubled grid
  float frac;      // 2^-sh
  float sscale;    // s = GU * sscale
  int N;
  int shift_x, shift_y;  // N/2 - x0, N/2 - y0: the sum is taken about the image's middle
  float coef[kTaps / 2][2 * kPolyHalf];
};

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// The 8 taps of the spreading kernel at cell fraction f: tap t is the kernel
// at distance f + 3 - t.  Tap 7 - t is tap t mirrored, so even and odd parts
// of one polynomial in f - 1/2 give both.
__device__ __forceinline__ void taps(const SpreadArgs& a, float f, float (&w)[kTaps]) {
  const float z = f - 0.5f, z2 = z * z;
#pragma unroll
  for (int t = 0; t < kTaps / 2; t++) {
    float e = a.coef[t][kPolyHalf - 1], o = a.coef[t][2 * kPolyHalf - 1];
#pragma unroll
    for (int k = kPolyHalf - 2; k >= 0; k--) {
      e = fmaf(e, z2, a.coef[t][k]);
      o = fmaf(o, z2, a.coef[t][kPolyHalf + k]);
    }
    w[t] = fmaf(o, z, e);
    w[kTaps - 1 - t] = fmaf(-o, z, e);
  }
}

// One warp per task.  Each lane prepares one of 32 visibilities at a time
// (position, taps, the pairs' values) in shared memory; then the warp takes
// them one by one, lane l summing taps (l & 7, l >> 3) and (l & 7, 4 + l >> 3)
// of every plane in registers as long as the first cell stays the same (the
// visibilities are sorted by cell), and adds them to the task's 15 x 15 tile
// in shared memory when it changes.  The tile goes out once, to the task's
// own slot, so no two warps write the same place.
template <int NP>
__global__ void __launch_bounds__(32 * kSpreadWarps) k_nu_spread(SpreadArgs a) {
  extern __shared__ float4 smem_f4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPerWarp = NP * kTilePts + NP * 32 + 32 * 5;  // float4
  float4* tile = smem_f4 + warp * kPerWarp;
  float4* val = tile + NP * kTilePts;           // [NP][32]
  float* wts = reinterpret_cast<float*>(val + NP * 32);  // [32][20]: x taps, y taps, padding
  const int id = blockIdx.x * kSpreadWarps + warp;
  if (id >= a.ntasks) return;
  const NuTask task = a.tasks[id];
  for (int k = lane; k < NP * kTilePts; k += 32) tile[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int tx = lane & 7, ty = lane >> 3;
  f32x2 acc[2][NP][2];
  auto clear = [&]() {
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int q = 0; q < NP; q++) acc[h][q][0] = acc[h][q][1] = 0ull;
  };
  auto flush = [&](int base) {
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int idx = base + (ty + 4 * h) * kTileSide + tx;
#pragma unroll
      for (int q = 0; q < NP; q++) {
        float4 t = tile[q * kTilePts + idx];
        const float2 p = unpack2(acc[h][q][0]), m = unpack2(acc[h][q][1]);
        t.x += p.x;
        t.y += p.y;
        t.z += m.x;
        t.w += m.y;
        tile[q * kTilePts + idx] = t;
      }
    }
  };
  clear();
  int cur = -1;
  for (int k0 = 0; k0 < task.count; k0 += 32) {
    const int cnt = min(32, task.count - k0);
    __syncwarp();  // the last 32 are done with the staging
    int base = 0;
    if (lane < cnt) {
      const uint32_t g = task.begin + k0 + lane;
      const uint4 p = __ldcs(a.ph + g);
      float2 c;
      if (a.mode <= 1 || a.mode == 4) {
        c = __ldcs(a.cvr + g);
        if (a.mode == 4) c.y = -c.y;
      } else {
        const float w = a.deg[g].w;
        if (a.mode == 3) {
          c = make_float2(w, 0.0f);
        } else {
          const float2 o = a.vo[g];
          c = make_float2(w * o.x, w * o.y);
        }
      }
      // fold into u >= 0: Re(conj(c) e^{i t}) = Re(c e^{-i t})
      const bool neg = p.x >> 31;
      const uint32_t fu = neg ? 0u - p.x : p.x, fv = neg ? 0u - p.y : p.y;
      float2 v = make_float2(c.x, neg ? c.y : -c.y);
      float s = __uint_as_float(p.z) * a.sscale;
      if (neg) s = -s;
      if (a.shift_x | a.shift_y) {
        const uint32_t t = (uint32_t)a.shift_x * fu + (uint32_t)a.shift_y * fv;
        float sn, cs;
        sincospif((float)(int32_t)t * 4.656612873077393e-10f, &sn, &cs);
        v = make_float2(v.x * cs - v.y * sn, v.x * sn + v.y * cs);
      }
      const uint32_t below = (1u << a.sh) - 1u;
      const int ix = (int)(fu >> a.sh), iy = (int)((int32_t)fv >> a.sh) + a.N;
      base = (iy & 7) * kTileSide + (ix & 7);
      float w[kTaps];
      float4* wl = reinterpret_cast<float4*>(wts + lane * 20);
      taps(a, (float)(fu & below) * a.frac, w);
      wl[0] = make_float4(w[0], w[1], w[2], w[3]);
      wl[1] = make_float4(w[4], w[5], w[6], w[7]);
      taps(a, (float)(fv & below) * a.frac, w);
      wl[2] = make_float4(w[0], w[1], w[2], w[3]);
      wl[3] = make_float4(w[4], w[5], w[6], w[7]);
      float te = 1.0f, to = s;  // T_2q, T_2q+1
#pragma unroll
      for (int q = 0; q < NP; q++) {
        const float tp = te + to, tm = te - to;
        val[q * 32 + lane] = make_float4(v.x * tp, v.y * tp, v.x * tm, v.y * tm);
        te = fmaf(2.0f * s, to, -te);
        to = fmaf(2.0f * s, te, -to);
      }
    }
    int prev = __shfl_up_sync(0xffffffffu, base, 1);
    if (lane == 0) prev = cur;
    const uint32_t heads = __ballot_sync(0xffffffffu, base != prev);
    __syncwarp();
#pragma unroll 2
    for (int i = 0; i < cnt; i++) {
      if ((heads >> i) & 1u) {
        if (cur >= 0) {
          flush(cur);
          clear();
        }
        cur = __shfl_sync(0xffffffffu, base, i);
      }
      const float kx = wts[i * 20 + tx];
      const float w0 = kx * wts[i * 20 + 8 + ty], w1 = kx * wts[i * 20 + 12 + ty];
      const f32x2 p0 = pack2(w0, w0), p1 = pack2(w1, w1);
#pragma unroll
      for (int q = 0; q < NP; q++) {
        const float4 v = val[q * 32 + i];
        const f32x2 vp = pack2(v.x, v.y), vm = pack2(v.z, v.w);
        acc[0][q][0] = fma2(p0, vp, acc[0][q][0]);
        acc[0][q][1] = fma2(p0, vm, acc[0][q][1]);
        acc[1][q][0] = fma2(p1, vp, acc[1][q][0]);
        acc[1][q][1] = fma2(p1, vm, acc[1][q][1]);
      }
    }
  }
  if (cur >= 0) flush(cur);
  __syncwarp();
  float2* out = a.slots + (size_t)id * (NP * 2 * kTilePts);
  for (int k = lane; k < kTilePts; k += 32) {
#pragma unroll
    for (int q = 0; q < NP; q++) {
      const float4 t = tile[q * kTilePts + k];
      out[(2 * q) * kTilePts + k] = make_float2(t.x, t.y);
      out[(2 * q + 1) * kTilePts + k] = make_float2(t.z, t.w);
    }
  }
}

struct MergeArgs {
  const float2* __restrict__ slots;
  const int* __restrict__ slot_off;
  float2* __restrict__ F;
  int N, pairs, c0, t0;  // first channel and first task of the group
  int cmin, ncol, rmin, nrow, wrap;
  int tx0, ntx, ty0, nty;
};

// Sum of a plane at (column c, row r) over the tiles whose footprint holds
// it (two per axis at most) and their tasks, in order.
__device__ __forceinline__ float2 plane_at(const MergeArgs& a, int ch, int plane, int c, int r) {
  float2 s = make_float2(0.0f, 0.0f);
  const int cc = c + 3, rr = r + a.N + 3;
  if (cc < 0 || rr < 0) return s;
#pragma unroll
  for (int dy = 0; dy < 2; dy++) {
    const int ty = (rr >> 3) - dy - a.ty0, ly = (rr & 7) + 8 * dy;
    if (ly >= kTileSide || (unsigned)ty >= (unsigned)a.nty) continue;
#pragma unroll
    for (int dx = 0; dx < 2; dx++) {
      const int tx = (cc >> 3) - dx - a.tx0, lx = (cc & 7) + 8 * dx;
      if (lx >= kTileSide || (unsigned)tx >= (unsigned)a.ntx) continue;
      const int* so = a.slot_off + ((size_t)ch * a.nty + ty) * a.ntx + tx;
      const int s0 = __ldg(so) - a.t0, s1 = __ldg(so + 1) - a.t0;
      const float2* p = a.slots + ((size_t)s0 * a.pairs * 2 + plane) * kTilePts +
                        ly * kTileSide + lx;
      for (int k = s0; k < s1; k++, p += (size_t)a.pairs * 2 * kTilePts) {
        const float2 v = *p;
        s.x += v.x;
        s.y += v.y;
      }
    }
  }
  return s;
}

// F = (h+ (c, r) + conj(h- (-c, -r))) / 2 with h+- the sums of the even plus /
// minus the odd term: the Hermitian part of the even term's grid plus the
// anti-Hermitian part of the odd one's.
__global__ void __launch_bounds__(128) k_nu_merge(MergeArgs a) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= a.ncol) return;
  const int c = a.cmin + ci, r = a.rmin + blockIdx.y;
  const int ch = a.c0 + blockIdx.z / a.pairs, q = blockIdx.z % a.pairs;
  float2 hp = make_float2(0.0f, 0.0f), hm = hp;
  const int G = 2 * a.N;
  const int w = a.wrap ? 1 : 0;
  for (int wy = -w; wy <= w; wy++)
    for (int wx = -w; wx <= w; wx++) {
      const int cc = c + wx * G, rr = r + wy * G;
      const float2 p = plane_at(a, ch, 2 * q, cc, rr);
      const float2 m = plane_at(a, ch, 2 * q + 1, -cc, -rr);
      hp.x += p.x;
      hp.y += p.y;
      hm.x += m.x;
      hm.y += m.y;
    }
  a.F[((size_t)blockIdx.z * a.nrow + blockIdx.y) * a.ncol + ci] =
      make_float2(0.5f * (hp.x + hm.x), 0.5f * (hp.y - hm.y));
}

// An inverse FFT over the 2N cells of a line, of which the N outputs about
// the middle are kept: X[x] = E[x mod N] + e^{2 pi i x / 2N} O[x mod N] with
// the N-point transforms E, O of the even and odd cells.
template <int VPT>
__global__ void __launch_bounds__(VPT == 16 ? 512 : 256) k_nu_rows(
    int N, int log2n, int cmin, int ncol, int nrow, const float2* __restrict__ F,
    const float2* __restrict__ tw, const float2* __restrict__ turn, float2* __restrict__ H) {
  extern __shared__ float2 buf[];
  const float2* f = F + ((size_t)blockIdx.y * nrow + blockIdx.x) * ncol;
  const int stride = fft_stride(N);
  float2 v[VPT];
#pragma unroll
  for (int k = 0; k < VPT; k++) {
    const int p = threadIdx.x + k * blockDim.x;
    const int c = (p < N ? p : p - 2 * N) - cmin;
    v[k] = (p < 2 * N && (unsigned)c < (unsigned)ncol) ? f[c] : make_float2(0.0f, 0.0f);
  }
#pragma unroll
  for (int k = 0; k < VPT; k++) {
    const int p = threadIdx.x + k * blockDim.x;
    if (p < 2 * N) buf[(p & 1) * stride + fpad(p >> 1)] = v[k];
  }
  __syncthreads();
  smem_fft<VPT>(buf, log2n, 2, tw);
  float2* h = H + ((size_t)blockIdx.y * nrow + blockIdx.x) * N;
  for (int j = threadIdx.x; j < N; j += blockDim.x) {
    const int m = (j + N / 2) & (N - 1);
    const float2 e = buf[fpad(m)], o = cmul(buf[stride + fpad(m)], __ldg(turn + j));
    h[j] = make_float2(e.x + o.x, e.y + o.y);
  }
}

// The factor of every pixel's sum for one channel (blockIdx.y): beam,
// fg_scale, GCF and the chain rule as the direct engines apply them, 0
// outside the mask.
struct FactorArgs {
  int N, c0;
  int64_t MN;
  int mode, flag_opt, normalize, pb;
  float nu_0, D, pbf, pbcut, fg_scale, threshold;
  const float* __restrict__ beam_x;
  const float* __restrict__ beam_y;
  const float* __restrict__ chfreq;
  const int64_t* __restrict__ chnvis;
  const uint8_t* __restrict__ mask;
  const float* __restrict__ img;
  const float* __restrict__ gcf;
  float* __restrict__ fac;
};

__global__ void __launch_bounds__(256) k_nu_factors(FactorArgs a) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= a.MN) return;
  const int c = a.c0 + blockIdx.y;
  float f = 0.0f;
  if (a.mask[q] & kMaskIn) {
    const int i = (int)(q / a.N), j = (int)(q - (int64_t)i * a.N);
    const float freq = a.chfreq[c];
    f = -(a.fg_scale *
          attenuation_xy(a.beam_x[j], a.beam_y[i], freq, a.D, a.pbf, a.pbcut, a.pb));
    if (a.gcf) f *= a.gcf[q];
    if (a.normalize) f /= (float)a.chnvis[c];
    if (a.mode == 0) {
      const float nudiv = freq / a.nu_0;
      const float al = a.img[a.MN + q];
      const float pw = al == 0.0f ? 1.0f : powf(nudiv, al);
      if (a.flag_opt % 2 == 0) {
        f *= pw;
      } else {
        const float i0 = a.img[q];
        f = i0 > a.threshold ? f * (i0 * pw * a.fg_scale * logf(nudiv)) : 0.0f;
      }
    }
  }
  a.fac[blockIdx.y * a.MN + q] = f;
}

// Per pixel and pair the w-term's coefficients of the transform's real and
// imaginary parts, 2 (-1)^q J_2q(a) (J_0 once) and -2 (-1)^q J_2q+1(a), times
// the spreading kernel's correction.  Fixed by the geometry: made once.
__device__ __forceinline__ float bessel_tail(float h2, int n) {  // J_n(2h) n! / h^n, h <= 0.53
  float r = 1.0f - h2 / (5.0f * (n + 5));
  r = 1.0f - h2 / (4.0f * (n + 4)) * r;
  r = 1.0f - h2 / (3.0f * (n + 3)) * r;
  r = 1.0f - h2 / (2.0f * (n + 2)) * r;
  return 1.0f - h2 / (float)(n + 1) * r;
}

__global__ void __launch_bounds__(256) k_nu_coefficients(int N, int pairs, float wscale,
                                                         const float* __restrict__ beam_x,
                                                         const float* __restrict__ beam_y,
                                                         const float* __restrict__ corr,
                                                         float2* __restrict__ coef) {
  const int64_t px = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, MN = (int64_t)N * N;
  if (px >= MN) return;
  const int i = (int)(px / N), j = (int)(px - (int64_t)i * N);
  const float x = beam_x[j], y = beam_y[i], r2 = fmaf(x, x, y * y);
  // a / 2, a = wscale (z - 1)
  const float h = -0.5f * wscale * (r2 / (1.0f + sqrtf(1.0f - r2))), h2 = h * h;
  float p = corr[i] * corr[j];
  for (int q = 0; q < pairs; q++) {
    const float c = (q ? 2.0f : 1.0f) * (q & 1 ? -1.0f : 1.0f);
    const float ke = c * p * bessel_tail(h2, 2 * q);
    p *= h / (float)(2 * q + 1);
    const float ko = (q & 1 ? 2.0f : -2.0f) * p * bessel_tail(h2, 2 * q + 1);
    p *= h / (float)(2 * q + 2);
    coef[q * MN + px] = make_float2(ke, ko);
  }
}

struct ColArgs {
  int N, log2n, lcb;  // 2^lcb columns per block
  int64_t MN;
  int nchan;          // channels of the group
  int rmin, nrow;
  int wterm;
  const float2* __restrict__ H;
  const float2* __restrict__ tw;
  const float2* __restrict__ turn;
  const float* __restrict__ corr;
  const float2* __restrict__ coef;  // [pair][MN]
  const float* __restrict__ fac;    // [channel of the group][MN], or null: 1
  const uint8_t* __restrict__ mask; // pixels written (kMaskIn), or null: all
  float* __restrict__ out;
};

template <int VPT, int NP>
__global__ void __launch_bounds__(VPT == 16 ? 512 : 256, VPT == 16 ? 1 : 4) k_nu_cols(ColArgs a) {
  extern __shared__ float2 buf[];
  const int N = a.N, cb = 1 << a.lcb, j0 = blockIdx.x << a.lcb;
  const int stride = fft_stride(N);
  float acc[VPT / 2];
#pragma unroll
  for (int k = 0; k < VPT / 2; k++) acc[k] = 0.0f;
  for (int c = 0; c < a.nchan; c++) {
#pragma unroll 1
    for (int q = 0; q < NP; q++) {
      {
        const float2* h = a.H + (size_t)(c * NP + q) * a.nrow * N + j0;
        float2 v[VPT];
#pragma unroll
        for (int k = 0; k < VPT; k++) {
          const int idx = threadIdx.x + k * blockDim.x;
          const int p = idx >> a.lcb;
          const int r = (p < N ? p : p - 2 * N) - a.rmin;
          v[k] = (p < 2 * N && (unsigned)r < (unsigned)a.nrow)
                     ? h[(size_t)r * N + (idx & (cb - 1))]
                     : make_float2(0.0f, 0.0f);
        }
        __syncthreads();  // the last transform has been read
#pragma unroll
        for (int k = 0; k < VPT; k++) {
          const int idx = threadIdx.x + k * blockDim.x;
          const int p = idx >> a.lcb;
          if (p < 2 * N) buf[(2 * (idx & (cb - 1)) + (p & 1)) * stride + fpad(p >> 1)] = v[k];
        }
      }
      __syncthreads();
      smem_fft<VPT>(buf, a.log2n, 2 * cb, a.tw);
#pragma unroll
      for (int k = 0; k < VPT / 2; k++) {
        const int idx = threadIdx.x + k * blockDim.x;
        const int i = idx >> a.lcb, cc = idx & (cb - 1);
        if (i >= N) continue;
        const int64_t px = (int64_t)N * i + j0 + cc;
        const int m = fpad((i + N / 2) & (N - 1));
        const float2 e = buf[2 * cc * stride + m];
        const float2 o = cmul(buf[(2 * cc + 1) * stride + m], __ldg(a.turn + i));
        float t;
        if (a.wterm) {
          const float2 kk = __ldg(a.coef + q * a.MN + px);
          t = fmaf(kk.x, e.x + o.x, kk.y * (e.y + o.y));
        } else {
          t = q == 0 ? (e.x + o.x) * (__ldg(a.corr + i) * __ldg(a.corr + j0 + cc)) : 0.0f;
        }
        acc[k] = fmaf(a.fac ? __ldg(a.fac + c * a.MN + px) : 1.0f, t, acc[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < VPT / 2; k++) {
    const int idx = threadIdx.x + k * blockDim.x;
    const int i = idx >> a.lcb;
    if (i >= N) continue;
    const int64_t px = (int64_t)N * i + j0 + (idx & (cb - 1));
    if (!a.mask || (a.mask[px] & kMaskIn)) a.out[px] += acc[k];
  }
}

// ---- plan ------------------------------------------------------------------

// first visibility of each (channel, tile) among the sorted, kept ones
__global__ void k_tile_heads(int64_t n, const unsigned long long* __restrict__ keys,
                             int* __restrict__ head) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const unsigned long long key = keys[k];
  const bool kept = (uint32_t)key != 0xFFFFFFFFu;
  head[k] = kept && (k == 0 || (keys[k - 1] >> 6) != (key >> 6)) ? 1 : 0;
}

__global__ void k_tile_runs(int64_t n, const unsigned long long* __restrict__ keys,
                            const int* __restrict__ head, const int* __restrict__ pos,
                            unsigned long long* __restrict__ run_key,
                            uint32_t* __restrict__ run_start) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n || !head[k]) return;
  run_key[pos[k]] = keys[k] >> 6;
  run_start[pos[k]] = (uint32_t)k;
}

double kernel_value(double z) {
  const double t = 2.0 * z / kTaps;
  return std::fabs(t) < 1.0 ? std::exp(kBeta * (std::sqrt(1.0 - t * t) - 1.0)) : 0.0;
}

// The taps' polynomials: Chebyshev interpolation of degree 11 over the cell,
// even and odd coefficients in f - 1/2 apart.
void tap_polynomials(float (&coef)[kTaps / 2][2 * kPolyHalf]) {
  constexpr int D = 2 * kPolyHalf;
  for (int t = 0; t < kTaps / 2; t++) {
    double cheb[D] = {0.0};
    for (int m = 0; m < D; m++)
      for (int k = 0; k < D; k++) {
        const double th = kPiD * (k + 0.5) / D;
        cheb[m] += (m ? 2.0 : 1.0) / D * std::cos(m * th) *
                   kernel_value(0.5 * std::cos(th) + 3.5 - t);
      }
    // to powers of y = 2 (f - 1/2), then of f - 1/2
    double pw[D] = {0.0}, a[D] = {1.0}, b[D] = {0.0, 1.0};  // T_0, T_1
    for (int m = 0; m < D; m++) {
      for (int k = 0; k < D; k++) pw[k] += cheb[m] * a[k];
      double nx[D];
      for (int k = 0; k < D; k++) nx[k] = (k ? 2.0 * b[k - 1] : 0.0) - a[k];
      for (int k = 0; k < D; k++) {
        a[k] = b[k];
        b[k] = nx[k];
      }
    }
    for (int k = 0; k < D; k++)
      coef[t][(k & 1) * kPolyHalf + k / 2] = (float)std::ldexp(pw[k], k);
  }
}

// 1 / the kernel's Fourier transform at x / 2N cycles per cell, by the
// trapezoidal rule (the kernel falls smoothly to e^-beta at its ends).
std::vector<float> kernel_correction(int N) {
  constexpr int S = 16 * kTaps;  // steps over half the support
  double val[S];
  for (int k = 0; k < S; k++) val[k] = (k ? 1.0 : 0.5) * kernel_value(kTaps / 2.0 * k / S);
  std::vector<float> c(N);
  for (int j = 0; j <= N / 2; j++) {
    const double xi = (double)(j - N / 2) / (2.0 * N);
    double s = 0.0;
    for (int k = 0; k < S; k++) s += val[k] * std::cos(2.0 * kPiD * xi * (kTaps / 2.0 * k / S));
    c[j] = (float)(1.0 / (2.0 * s * (kTaps / 2.0) / S));
  }
  for (int j = N / 2 + 1; j < N; j++) c[j] = c[N - j];
  return c;
}

template <int NP>
gv_status spread(const SpreadArgs& a, cudaStream_t st) {
  const size_t smem =
      sizeof(float4) * kSpreadWarps * (size_t)(NP * kTilePts + NP * 32 + 32 * 5);
  if (smem > 48 * 1024)
    GV_CUDA(cudaFuncSetAttribute(k_nu_spread<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_nu_spread<NP><<<(a.ntasks + kSpreadWarps - 1) / kSpreadWarps, 32 * kSpreadWarps, smem, st>>>(a);
  GV_LAUNCH("k_nu_spread");
  return GV_OK;
}

template <int VPT>
gv_status rows(const Problem& P, const NuPlan& n, int nplanes, int threads, const float2* tw) {
  const size_t smem = sizeof(float2) * 2 * fft_stride(P.N);
  if (smem > 48 * 1024)
    GV_CUDA(cudaFuncSetAttribute(k_nu_rows<VPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_nu_rows<VPT><<<dim3(n.nrow, nplanes), threads, smem, P.stream>>>(
      P.N, P.log2n, n.cmin, n.ncol, n.nrow, n.d_F, tw, n.d_turn, n.d_H);
  GV_LAUNCH("k_nu_rows");
  return GV_OK;
}

template <int VPT, int NP>
gv_status cols(const ColArgs& a, int threads, cudaStream_t st) {
  const size_t smem = sizeof(float2) * (size_t)(2 << a.lcb) * fft_stride(a.N);
  if (smem > 48 * 1024)
    GV_CUDA(cudaFuncSetAttribute(k_nu_cols<VPT, NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_nu_cols<VPT, NP><<<a.N >> a.lcb, threads, smem, st>>>(a);
  GV_LAUNCH("k_nu_cols");
  return GV_OK;
}

template <int VPT>
gv_status cols_pairs(int pairs, const ColArgs& a, int threads, cudaStream_t st) {
  switch (pairs) {
    case 1: return cols<VPT, 1>(a, threads, st);
    case 2: return cols<VPT, 2>(a, threads, st);
    case 3: return cols<VPT, 3>(a, threads, st);
    default: return cols<VPT, 4>(a, threads, st);
  }
}

// largest |z - 1| over the image
double max_depth(const Problem& P) {
  const double hx = std::max(std::fabs((double)(0 - (int)P.xobs)),
                             std::fabs((double)(P.M - 1 - (int)P.xobs))) * std::fabs(P.dx_rad);
  const double hy = std::max(std::fabs((double)(0 - (int)P.yobs)),
                             std::fabs((double)(P.N - 1 - (int)P.yobs))) * std::fabs(P.dy_rad);
  const double r2 = hx * hx + hy * hy;
  return r2 < 1.0 ? r2 / (1.0 + std::sqrt(1.0 - r2)) : 1.0;
}

}  // namespace

void nu_free(Problem& P) {
  if (!P.nu) return;
  NuPlan* n = P.nu;
  cudaFree(n->d_tasks);
  cudaFree(n->d_slot_off);
  cudaFree(n->d_slots);
  cudaFree(n->d_F);
  cudaFree(n->d_H);
  cudaFree(n->d_turn);
  cudaFree(n->d_corr);
  cudaFree(n->d_coef);
  cudaFree(n->d_fac);
  delete n;
  P.nu = nullptr;
}

// The pixels' w-term coefficients, once the beam tables (the pixels' offsets)
// are in place.
gv_status nu_finish(Problem& P) {
  if (!P.nu) return GV_OK;
  const NuPlan& n = *P.nu;
  const int64_t MN = (int64_t)P.N * P.N;
  k_nu_coefficients<<<(unsigned)((MN + 255) / 256), 256, 0, P.stream>>>(
      P.N, n.pairs, (float)(2.0 * kPiD * n.wmax), P.d_beam_x, P.d_beam_y, n.d_corr, n.d_coef);
  GV_LAUNCH("k_nu_coefficients");
  return GV_OK;
}

uint32_t nu_tiles_x(int N) { return (uint32_t)(N / 8 + 1); }

// Builds the plan of P (P.nu stays null where the direct sums are to run):
// keys are the sorted (channel << 32 | tile << 6 | cell in tile) of all
// visibilities, all ones in the low word for those left out.
gv_status nu_setup(Problem& P, const unsigned long long* d_keys, double maxw) {
  const int C = (int)P.chans.size(), N = P.N;
  if (P.Vgrid <= 0 || P.V >= (int64_t(1) << 31)) return GV_OK;
  const double A = 2.0 * kPiD * maxw * max_depth(P);
  int pairs = 1;
  auto left = [&](int np) {
    double t = 2.0;
    for (int k = 1; k <= 2 * np; k++) t *= 0.5 * A / k;
    return t;
  };
  while (pairs <= kMaxPairs && left(pairs) > kWTol) pairs++;
  if (pairs > kMaxPairs) return GV_OK;
  cudaStream_t st = P.stream;
  // ---- runs of visibilities of one tile -------------------------------------
  std::vector<unsigned long long> rkey;
  std::vector<uint32_t> rstart;
  {
    const int64_t V = P.V;
    int *head = nullptr, *pos = nullptr;
    void* tmp = nullptr;
    unsigned long long* dk = nullptr;
    uint32_t* ds = nullptr;
    const size_t tb = scan_scratch(V);
    auto work = [&]() -> gv_status {
      GV_CUDA(cudaMalloc(&head, sizeof(int) * V));
      GV_CUDA(cudaMalloc(&pos, sizeof(int) * V));
      GV_CUDA(cudaMalloc(&tmp, tb));
      const unsigned gb = (unsigned)((V + 255) / 256);
      k_tile_heads<<<gb, 256, 0, st>>>(V, d_keys, head);
      GV_LAUNCH("k_tile_heads");
      GV_TRY(exclusive_scan<int>(tmp, tb, head, pos, V, st));
      int last[2] = {0, 0};
      GV_CUDA(cudaMemcpyAsync(&last[0], head + V - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
      GV_CUDA(cudaMemcpyAsync(&last[1], pos + V - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
      GV_CUDA(cudaStreamSynchronize(st));
      const size_t R = (size_t)last[0] + last[1];
      rkey.resize(R);
      rstart.resize(R);
      GV_CUDA(cudaMalloc(&dk, sizeof(*dk) * R));
      GV_CUDA(cudaMalloc(&ds, sizeof(*ds) * R));
      k_tile_runs<<<gb, 256, 0, st>>>(V, d_keys, head, pos, dk, ds);
      GV_LAUNCH("k_tile_runs");
      GV_CUDA(cudaMemcpyAsync(rkey.data(), dk, sizeof(*dk) * R, cudaMemcpyDeviceToHost, st));
      GV_CUDA(cudaMemcpyAsync(rstart.data(), ds, sizeof(*ds) * R, cudaMemcpyDeviceToHost, st));
      GV_CUDA(cudaStreamSynchronize(st));
      return GV_OK;
    };
    const gv_status s = work();
    cudaFree(head);
    cudaFree(pos);
    cudaFree(tmp);
    cudaFree(dk);
    cudaFree(ds);
    if (s != GV_OK) return s;
  }
  const size_t R = rkey.size();
  const uint32_t NTX = nu_tiles_x(N);
  NuPlan* n = new NuPlan();
  P.nu = n;
  n->pairs = pairs;
  n->wmax = (float)(maxw > 0.0 ? maxw : 1.0);
  // tiles in use
  int txa = 1 << 30, txb = -1, tya = 1 << 30, tyb = -1;
  for (size_t r = 0; r < R; r++) {
    const uint32_t t = (uint32_t)(rkey[r] & 0x3FFFFFFu);
    const int tx = (int)(t % NTX), ty = (int)(t / NTX);
    txa = std::min(txa, tx);
    txb = std::max(txb, tx);
    tya = std::min(tya, ty);
    tyb = std::max(tyb, ty);
  }
  n->tx0 = txa;
  n->ntx = txb - txa + 1;
  n->ty0 = tya;
  n->nty = tyb - tya + 1;
  // covered cells: footprints are columns 8 tx - 3 .. 8 tx + 11, rows
  // 8 ty - N - 3 .. 8 ty - N + 11, and their mirror images
  const int cmax = 8 * txb + 11, rlo = 8 * tya - N - 3, rhi = 8 * tyb - N + 11;
  const int rmax = std::max(rhi, -rlo);
  n->wrap = cmax > N - 1 || rmax > N - 1;
  n->cmin = n->wrap ? -N : -cmax;
  n->ncol = n->wrap ? 2 * N : (2 * cmax + 1 + 1) & ~1;
  n->rmin = n->wrap ? -N : -rmax;
  n->nrow = n->wrap ? 2 * N : 2 * rmax + 1;
  // ---- tasks ------------------------------------------------------------------
  // a tile's visibilities in pieces of T: enough pieces to fill the GPU (32
  // warps per SM) without more slots than the sums are worth
  const int64_t want = P.Vgrid / std::max(1, 32 * P.num_sms);
  const int T = (int)std::min<int64_t>(1024, std::max<int64_t>(32, want / 32 * 32));
  std::vector<NuTask> tasks;
  const size_t tiles = (size_t)n->nty * n->ntx;
  std::vector<int> off((size_t)C * tiles + 1, 0);
  n->task_off.assign(C + 1, 0);
  for (size_t r = 0; r < R; r++) {
    const uint32_t t = (uint32_t)(rkey[r] & 0x3FFFFFFu);
    const int c = (int)(rkey[r] >> 26);
    const int64_t end_c = P.chans[c].off + P.chans[c].ngrid;
    const int64_t end = (r + 1 < R && (int)(rkey[r + 1] >> 26) == c) ? rstart[r + 1] : end_c;
    const int64_t cnt = end - rstart[r];
    const int parts = (int)((cnt + T - 1) / T);
    for (int k = 0; k < parts; k++) {
      const int64_t b = (int64_t)T * k;
      tasks.push_back({(uint32_t)(rstart[r] + b), (int)std::min<int64_t>(T, cnt - b)});
    }
    off[(size_t)c * tiles + (t / NTX - tya) * n->ntx + (t % NTX - txa) + 1] = parts;
    n->task_off[c + 1] += parts;
  }
  for (size_t k = 1; k < off.size(); k++) off[k] += off[k - 1];
  for (int c = 0; c < C; c++) n->task_off[c + 1] += n->task_off[c];
  // ---- channel groups whose workspace stays bounded ------------------------------
  const size_t slot_b = sizeof(float2) * 2 * kTilePts * pairs;
  const size_t f_b = sizeof(float2) * (size_t)pairs * n->nrow * n->ncol;
  const size_t h_b = sizeof(float2) * (size_t)pairs * n->nrow * N;
  const size_t fac_b = sizeof(float) * (size_t)N * N;
  n->groups.push_back(0);
  size_t max_slots = 0, max_ch = 0;
  for (int c = 0; c < C;) {
    size_t used = 0;
    const int c0 = c;
    while (c < C) {
      const size_t need = slot_b * (n->task_off[c + 1] - n->task_off[c]) + f_b + h_b + fac_b;
      if (c > c0 && used + need > kWorkspace) break;
      used += need;
      c++;
    }
    n->groups.push_back(c);
    max_ch = std::max<size_t>(max_ch, c - c0);
    max_slots = std::max<size_t>(max_slots, n->task_off[c] - n->task_off[c0]);
  }
  std::vector<float2> turn(N);
  for (int j = 0; j < N; j++) {
    const double t = kPiD * (j - N / 2) / N;
    turn[j] = make_float2((float)std::cos(t), (float)std::sin(t));
  }
  const std::vector<float> corr = kernel_correction(N);
  tap_polynomials(n->coef);
  auto upload = [&]() -> cudaError_t {
    cudaError_t e = cudaMalloc(&n->d_tasks, sizeof(NuTask) * tasks.size());
    if (e == cudaSuccess) e = cudaMalloc(&n->d_slot_off, sizeof(int) * off.size());
    if (e == cudaSuccess) e = cudaMalloc(&n->d_slots, slot_b * max_slots);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_F, f_b * max_ch);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_H, h_b * max_ch);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_turn, sizeof(float2) * N);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_corr, sizeof(float) * N);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_coef, sizeof(float2) * (size_t)pairs * N * N);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_fac, fac_b * max_ch);
    return e;
  };
  const cudaError_t e = upload();
  if (e == cudaErrorMemoryAllocation) {
    // no room for the grids: the direct sums need less
    cudaGetLastError();
    nu_free(P);
    return GV_OK;
  }
  if (e != cudaSuccess) return cuda_fail(e, "nu_setup");
  GV_CUDA(cudaMemcpy(n->d_tasks, tasks.data(), sizeof(NuTask) * tasks.size(),
                     cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemcpy(n->d_slot_off, off.data(), sizeof(int) * off.size(),
                     cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemcpy(n->d_turn, turn.data(), sizeof(float2) * N, cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemcpy(n->d_corr, corr.data(), sizeof(float) * N, cudaMemcpyHostToDevice));
  return GV_OK;
}

gv_status dchi2_nu(Problem& P, const float* d_img, int flag_opt, float* d_result,
                   int only_channel, int mode) {
  const NuPlan& n = *P.nu;
  const int N = P.N, np = n.pairs;
  SpreadArgs sa;
  sa.ph = P.d_ph;
  sa.cvr = P.d_cvr;
  sa.deg = P.d_deg;
  sa.vo = P.d_vo;
  sa.slots = n.d_slots;
  sa.mode = mode;
  sa.sh = 31 - P.log2n;
  sa.frac = std::ldexp(1.0f, -sa.sh);
  sa.sscale = (float)(2.0 / (P.dx_rad * P.dx_rad) / n.wmax);
  sa.N = N;
  sa.shift_x = N / 2 - (int)P.xobs;
  sa.shift_y = N / 2 - (int)P.yobs;
  std::copy(&n.coef[0][0], &n.coef[0][0] + sizeof(n.coef) / sizeof(float), &sa.coef[0][0]);
  MergeArgs ma;
  ma.slots = n.d_slots;
  ma.slot_off = n.d_slot_off;
  ma.F = n.d_F;
  ma.N = N;
  ma.pairs = np;
  ma.cmin = n.cmin;
  ma.ncol = n.ncol;
  ma.rmin = n.rmin;
  ma.nrow = n.nrow;
  ma.wrap = n.wrap;
  ma.tx0 = n.tx0;
  ma.ntx = n.ntx;
  ma.ty0 = n.ty0;
  ma.nty = n.nty;
  ColArgs ca;
  ca.N = N;
  ca.log2n = P.log2n;
  ca.MN = (int64_t)P.M * N;
  ca.rmin = n.rmin;
  ca.nrow = n.nrow;
  ca.H = n.d_H;
  ca.tw = P.d_twiddle;
  ca.turn = n.d_turn;
  ca.corr = n.d_corr;
  ca.wterm = mode == 4 ? 0 : 1;
  ca.coef = n.d_coef;
  ca.fac = mode <= 1 ? n.d_fac : nullptr;
  ca.mask = mode <= 1 ? P.d_mask : nullptr;
  ca.out = d_result + (mode == 0 ? (int64_t)(flag_opt % 2) * ca.MN : 0);
  FactorArgs fa;
  fa.N = N;
  fa.MN = ca.MN;
  fa.mode = mode;
  fa.flag_opt = flag_opt;
  fa.normalize = P.normalize;
  fa.pb = P.pb;
  fa.nu_0 = P.nu_0;
  fa.D = P.D;
  fa.pbf = P.pbf;
  fa.pbcut = P.pbcut;
  fa.fg_scale = P.fg_scale;
  fa.threshold = P.threshold;
  fa.beam_x = P.d_beam_x;
  fa.beam_y = P.d_beam_y;
  fa.chfreq = P.d_chfreq;
  fa.chnvis = P.d_chnvis;
  fa.mask = P.d_mask;
  fa.img = d_img;
  fa.gcf = P.d_gcf;
  fa.fac = n.d_fac;
  // columns per block: 256 blocks or more, 8192 values a block at most
  ca.lcb = N <= 256 ? 0 : (N == 512 ? 1 : (N == 1024 ? 2 : (N == 2048 ? 1 : 0)));
  std::vector<int> one = {only_channel, only_channel + 1};
  const std::vector<int>& groups = only_channel >= 0 ? one : n.groups;
  for (size_t g = 0; g + 1 < groups.size(); g++) {
    const int c0 = groups[g], c1 = groups[g + 1], nch = c1 - c0;
    const int t0 = n.task_off[c0];
    sa.tasks = n.d_tasks + t0;
    sa.ntasks = n.task_off[c1] - t0;
    if (sa.ntasks == 0) continue;
    switch (np) {
      case 1: GV_TRY(spread<1>(sa, P.stream)); break;
      case 2: GV_TRY(spread<2>(sa, P.stream)); break;
      case 3: GV_TRY(spread<3>(sa, P.stream)); break;
      default: GV_TRY(spread<4>(sa, P.stream)); break;
    }
    ma.c0 = c0;
    ma.t0 = t0;
    k_nu_merge<<<dim3((n.ncol + 127) / 128, n.nrow, nch * np), 128, 0, P.stream>>>(ma);
    GV_LAUNCH("k_nu_merge");
    if (N <= 256) GV_TRY(rows<2>(P, n, nch * np, 256, P.d_twiddle));
    else if (N == 512) GV_TRY(rows<4>(P, n, nch * np, 256, P.d_twiddle));
    else if (N == 1024) GV_TRY(rows<8>(P, n, nch * np, 256, P.d_twiddle));
    else GV_TRY(rows<16>(P, n, nch * np, N == 2048 ? 256 : 512, P.d_twiddle));
    if (mode <= 1) {
      fa.c0 = c0;
      k_nu_factors<<<dim3((unsigned)((ca.MN + 255) / 256), nch), 256, 0, P.stream>>>(fa);
      GV_LAUNCH("k_nu_factors");
    }
    ca.nchan = nch;
    if (N <= 256) GV_TRY(cols_pairs<2>(np, ca, 256, P.stream));
    else if (N == 512) GV_TRY(cols_pairs<8>(np, ca, 256, P.stream));
    else GV_TRY(cols_pairs<16>(np, ca, 512, P.stream));
  }
  return GV_OK;
}

}  // namespace gv
