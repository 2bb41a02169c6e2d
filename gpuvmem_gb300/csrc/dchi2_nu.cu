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
//  2. k_nu_rows    the tiles' sums added up along the rows of the grid that
//                  the data cover, and their FFTs, the image's N of 2N outputs;
//  3. k_nu_cols    column FFTs, the kernel's correction, the w-term, beam,
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
// All arithmetic is FP32 on exact 32-bit fixed-point grid positions, the sums
// over a tile's pieces and over the channels of a dirty image or PSF with their
// rounding errors kept; every sum is taken in a fixed order (no atomics), so
// results repeat bit for bit.  Against 64-bit sums gradients are 0.8 to 1.7e-7 off
// in the 2-norm (64^2 to 1024^2), where the tensor-core sum is 1.2 to 1.4e-6 off
// and the SIMT sum 0.8 to 2.7e-7; dirty images and PSFs 0.3 to 1.6e-7.  The
// kernel's truncation and the FFTs' rounding make that up, so it does not fall
// with the number of visibilities as the SIMT sum's error does where their terms
// add up (2.5e-8 for 2.1M visibilities of one 64^2 channel).
#include <algorithm>
#include <cmath>
#include <vector>

#include "fft.cuh"
#include "gv_internal.cuh"

namespace gv {

// Work of one block of k_nu_spread: `count` consecutive visibilities, all
// with their first cell in one 8 x 8 tile of the doubled grid.
struct NuTask {
  uint32_t begin;
  int count;
  int first, pieces;  // first task of the tile, tasks of the tile
};

struct NuPlan {
  int pairs = 0;           // complex FFTs per channel
  int warps = 1;           // of a block of k_nu_spread, or 8
  float wmax = 0.0f;
  int cmax = 0;            // covered columns: -cmax .. cmax
  int rmin = 0, nrow = 0;  // covered rows (signed)
  int wrap = 0;            // cells beyond +-N: the grid's period matters
  int tx0 = 0, ntx = 0, ty0 = 0, nty = 0;  // tiles in use
  std::vector<int> task_off;   // [C + 1]
  std::vector<int> groups;     // channel group boundaries
  NuTask* d_tasks = nullptr;
  int* d_slot = nullptr;       // [C nty ntx] first task of each tile, or -1
  // [tasks] tasks of a tile done (at its first task), [N] pieces of a column block done
  uint32_t* d_done = nullptr;
  int tasks = 0;
  float4* d_slots = nullptr;   // per task: [pair][225] sums {h+, h-}
  float2* d_H = nullptr;       // [channel of the group][pair][N / 4][nrow][4]
  float2* d_twiddle = nullptr; // fft16_twiddles(log2 2N)
  float* d_corr = nullptr;     // [N] 1 / kernel transform
  float2* d_coef = nullptr;    // [pair][MN] w-term coefficients (k_nu_coefficients)
  float* d_fac = nullptr;      // [C][MN] image-independent factors (k_nu_factors)
  float* d_part = nullptr;     // sums of shared column blocks, N >= 1024
  float coef[4][12];           // the taps' polynomials (tap_polynomials)
  // from nu_plan to nu_build
  std::vector<NuTask> h_tasks;
  std::vector<int> h_slot;
  size_t max_slots = 0, max_ch = 0;  // tasks and channels of the largest group
};

namespace {

constexpr int kTaps = 8;
constexpr int kTileSide = 15;  // 8 first cells + 7
constexpr int kTilePts = kTileSide * kTileSide;
constexpr int kMinShare = 16;  // visibilities a warp takes at least
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
  const NuTask* __restrict__ tasks;  // of the group
  int ntasks, t0;                    // t0: the group's first task
  uint32_t* __restrict__ done;
  float4* slots;
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

// s += x with the rounding error in e (Knuth's two-sum)
__device__ __forceinline__ void two_sum(float& s, float& e, float x) {
  const float t = s + x, b = t - s;
  e += (s - (t - b)) + (x - b);
  s = t;
}

// One block per task, its visibilities shared out among the warps in order.
// Each lane prepares one of 32 visibilities at a time (position, taps, the
// pairs' values) in shared memory; then the warp takes them one by one.  Lane
// l owns the cells whose column is l mod 8 and whose row is l / 8 or l / 8 + 4
// mod 8: of any 8 x 8 footprint exactly two, whose sums it keeps in registers
// while the footprint moves along a row of cells (the visibilities are sorted
// by cell), so a step to the next cell writes back only the column that is
// left.  The warps' 15 x 15 tiles are added in order and go out once, to the
// task's own slot; where a tile has several tasks, the last of their blocks
// to finish adds the slots up, in order and the sums of eight compensated (a
// dense tile has thousands of them), into the first.
//
// Bound by issue slots, two thirds of them at the 19 warps an SM that the tiles
// leave room for: 40 warp instructions a visibility.  8.8 M visibilities in 8
// channels, two pairs: 453 us (87 us of memory traffic; 563 with a test for a
// new cell at every visibility, whose loads then could not run ahead, and the
// two y taps read one by one).  Lanes four to a column, which writes a column
// back in fewer wavefronts: 3 % slower.
template <int NP, int kSpreadWarps>
__global__ void __launch_bounds__(32 * kSpreadWarps) k_nu_spread(SpreadArgs a) {
  extern __shared__ float4 smem_f4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kStage = NP * 32 + 32 * 5;  // float4 of a warp's staging
  float4* tile = smem_f4 + warp * (NP * kTilePts);
  float4* val = smem_f4 + kSpreadWarps * (NP * kTilePts) + warp * kStage;  // [NP][32]
  float* wts = reinterpret_cast<float*>(val + NP * 32);  // [32][20]: x taps, y taps, padding
  const NuTask task = a.tasks[blockIdx.x];
  // whole batches of 32, unless one would do for all the warps
  const int even = (task.count + kSpreadWarps - 1) / kSpreadWarps;
  const int share = kSpreadWarps == 1 ? task.count
                    : task.count <= 32 ? max(kMinShare, even) : (even + 31) & ~31;
  const int first = min(task.count, warp * share), last = min(task.count, first + share);
  const int tx = lane & 7, ty = lane >> 3;
  f32x2 acc[2][NP][2];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int q = 0; q < NP; q++) acc[h][q][0] = acc[h][q][1] = 0ull;
  // this lane's place in the footprint at (bx, by): its x tap and two y taps,
  // oy and oy + 4, which lie side by side in the staging
  int bx = 0, by = 0, ox = tx, oy = ty;
  auto flush = [&]() {
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int idx = (by + oy + 4 * h) * kTileSide + bx + ox;
#pragma unroll
      for (int q = 0; q < NP; q++) {
        float4 t = tile[q * kTilePts + idx];
        const float2 p = unpack2(acc[h][q][0]), m = unpack2(acc[h][q][1]);
        t.x += p.x;
        t.y += p.y;
        t.z += m.x;
        t.w += m.y;
        tile[q * kTilePts + idx] = t;
        acc[h][q][0] = acc[h][q][1] = 0ull;
      }
    }
  };
  if (first < last)
    for (int k = lane; k < NP * kTilePts; k += 32) tile[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  int cur = -1;
  for (int k0 = first; k0 < last; k0 += 32) {
    const int cnt = min(32, last - k0);
    __syncwarp();  // the last 32 are done with the staging
    int base = -1;
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
      base = ((iy & 7) << 3) | (ix & 7);
      float w[kTaps];
      float4* wl = reinterpret_cast<float4*>(wts + lane * 20);
      taps(a, (float)(fu & below) * a.frac, w);
      wl[0] = make_float4(w[0], w[1], w[2], w[3]);
      wl[1] = make_float4(w[4], w[5], w[6], w[7]);
      taps(a, (float)(fv & below) * a.frac, w);
      wl[2] = make_float4(w[0], w[4], w[1], w[5]);
      wl[3] = make_float4(w[2], w[6], w[3], w[7]);
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
    for (int i = 0; i < cnt;) {
      if ((heads >> i) & 1u) {
        const int next = __shfl_sync(0xffffffffu, base, i);
        const int nx = next & 7, ny = next >> 3;
        // every cell is one lane's, so the lanes that write back need not
        // wait for one another; the barrier orders one step after the last
        if (cur >= 0 && (ny != by || nx < bx || ox < nx - bx)) flush();
        __syncwarp();
        cur = next;
        bx = nx;
        by = ny;
        ox = (tx - bx) & 7;
        oy = (ty - by) & 3;
      }
      // the visibilities of this cell
      const uint32_t later = (heads >> i) & ~1u;
      const int end = later ? min(cnt, i + __ffs(later) - 1) : cnt;
#pragma unroll 4
      for (; i < end; i++) {
        const float kx = wts[i * 20 + ox];
        const float2 ky = *reinterpret_cast<const float2*>(wts + i * 20 + 8 + 2 * oy);
        const float w0 = kx * ky.x, w1 = kx * ky.y;
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
  }
  if (cur >= 0) flush();
  __syncthreads();
  const int nw = (task.count + share - 1) / share;
  constexpr size_t kSlot = NP * kTilePts;
  float4* out = a.slots + blockIdx.x * kSlot;
  for (int k = threadIdx.x; k < (int)kSlot; k += 32 * kSpreadWarps) {
    float4 t = smem_f4[k];
    for (int w = 1; w < nw; w++) {
      const float4 u = smem_f4[w * kSlot + k];
      t.x += u.x;
      t.y += u.y;
      t.z += u.z;
      t.w += u.w;
    }
    out[k] = t;
  }
  if (task.pieces == 1) return;
  __shared__ int last_block;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last_block = atomicAdd(a.done + task.first, 1u) == (uint32_t)task.pieces - 1u;
    if (last_block) a.done[task.first] = 0u;
  }
  __syncthreads();
  if (!last_block) return;
  __threadfence();
  float4* sum = a.slots + (size_t)(task.first - a.t0) * kSlot;
  for (int k = threadIdx.x; k < (int)kSlot; k += 32 * kSpreadWarps) {
    float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f), e = t;
    const float4* from = sum + k;
    for (int w = 0; w < task.pieces; w += 8, from += 8 * kSlot) {
      float4 u = __ldcg(from);
#pragma unroll
      for (int i = 1; i < 8; i++) {
        const float4 p = w + i < task.pieces ? __ldcg(from + i * kSlot)
                                             : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        u.x += p.x;
        u.y += p.y;
        u.z += p.z;
        u.w += p.w;
      }
      two_sum(t.x, e.x, u.x);
      two_sum(t.y, e.y, u.y);
      two_sum(t.z, e.z, u.z);
      two_sum(t.w, e.w, u.w);
    }
    sum[k] = make_float4(t.x + e.x, t.y + e.y, t.z + e.z, t.w + e.w);
  }
}

struct RowArgs {
  const float4* __restrict__ slots;
  const int* __restrict__ slot;
  const float2* __restrict__ tw;
  float2* __restrict__ H;
  int N, pairs, c0, t0;  // first channel and first task of the group
  int couples;           // (channel, pair, rows r and -r)
  int cmax, rmin, nrow, wrap;
  int tx0, ntx, ty0, nty;
};

// The tiles over a row of the grid (two at most) and the row's place in them.
struct RowTiles {
  const int* slot[2];
  int at[2];  // first cell of the row in the tile, or -1
};

__device__ __forceinline__ RowTiles row_tiles(const RowArgs& a, int ch, int r) {
  RowTiles t;
  const int rr = r + a.N + 3;
#pragma unroll
  for (int d = 0; d < 2; d++) {
    const int ty = (rr >> 3) - d - a.ty0, ly = (rr & 7) + 8 * d;
    const bool in = rr >= 0 && ly < kTileSide && (unsigned)ty < (unsigned)a.nty;
    t.slot[d] = a.slot + ((size_t)ch * a.nty + (in ? ty : 0)) * a.ntx;
    t.at[d] = in ? ly * kTileSide : -1;
  }
  return t;
}

// The sums {h+, h-} of pair q at column c of a row over the tiles that hold
// it, in order.
__device__ __forceinline__ float4 cell_at(const RowArgs& a, const RowTiles& t, int q, int c) {
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int cc = c + 3;
  const float4* p[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int tx = (cc >> 3) - (k & 1) - a.tx0, lx = (cc & 7) + 8 * (k & 1);
    int id = -1;
    if (cc >= 0 && lx < kTileSide && t.at[k >> 1] >= 0 && (unsigned)tx < (unsigned)a.ntx)
      id = __ldg(t.slot[k >> 1] + tx);
    p[k] = id >= 0 ? a.slots + ((size_t)(id - a.t0) * a.pairs + q) * kTilePts + t.at[k >> 1] + lx
                   : nullptr;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (p[k]) {
      const float4 v = __ldg(p[k]);
      s.x += v.x;
      s.y += v.y;
      s.z += v.z;
      s.w += v.w;
    }
  }
  return s;
}

// Rows r and -r of the doubled grid put together from the tiles and
// transformed over its 2N cells, of which the N outputs about the middle are
// kept: output x = j + r N / 8 of thread j is pixel x + N/2 for r < 4 and
// x - 2N + N/2 for r >= 12, so pixel j + s N / 8 is r = s - 4 or s + 12.
//
// The grid at (c, r) is (h+ (c, r) + conj(h- (-c, -r))) / 2, the Hermitian
// part of the even term's grid plus the anti-Hermitian part of the odd one's;
// the sums lie in u >= 0, so one cell of a tile feeds the two rows at c and
// -c.  Taking the rows together looks every cell up and reads it once.
// kPairs couples of rows per block.
//
// Bound by the waits between its phases (looking cells up, three exchanges)
// at two blocks an SM, about half of the issue slots: 16 planes of 2048^2 with
// 1223 covered rows, 372 us where its traffic takes 100 (381 with the registers
// that the rows beyond the grid's edge spilled); a row by itself, each cell
// looked up twice, 460.
template <int LG>
struct RowShape {
  static constexpr int kThreads = (1 << LG) / 16;  // per line
  static constexpr int kPairs = kThreads >= 64 ? 1 : 64 / kThreads;
  static constexpr int kBlock = 2 * kPairs * kThreads;
  static constexpr int kStride = span16(1 << LG);
  static constexpr size_t kSmem = sizeof(float2) * (2 * kPairs * kStride + kPairs * 14);
};

__device__ __forceinline__ constexpr int kept_output(int s) {
  return brev_c<4>(s < 4 ? s + 12 : s - 4);
}

template <int LG>
__global__ void __launch_bounds__(RowShape<LG>::kBlock, 1024 / RowShape<LG>::kBlock)
    k_nu_rows(RowArgs a) {
  using S = RowShape<LG>;
  constexpr int n = 1 << LG, N = n / 2, T = S::kThreads;
  extern __shared__ float2 smem_f2[];
  const int j = threadIdx.x % T, l = threadIdx.x / T;  // this thread's line: l & 1 of couple l / 2
  float2* buf = smem_f2 + l * S::kStride;
  const int couple = blockIdx.x * S::kPairs + (l >> 1);
  const bool in = couple < a.couples;
  // couple k of a plane: rows k and -k; 0 alone, or with -N where all rows are there
  const int per = a.wrap ? N : a.nrow / 2 + 1;
  const int plane = in ? couple / per : 0, k = in ? couple - plane * per : 0;
  const int ch = a.c0 + plane / a.pairs, q = plane % a.pairs;
  const int r = (l & 1) ? (k ? -k : -N) : k;
  const bool mine = in && (k > 0 || !(l & 1) || a.wrap);
  float2 v[16];
  if (!a.wrap) {
    // both lines' covered columns in the couple's two buffers (position c of
    // the transform), and h- of columns -3 .. 3, which meet h+ there
    float2* line0 = smem_f2 + (l & ~1) * S::kStride;
    float2* line1 = line0 + S::kStride;
    float2* near = smem_f2 + 2 * S::kPairs * S::kStride + (l >> 1) * 14;
    const int t = threadIdx.x % (2 * T);
    for (int p = t; p < n; p += 2 * T) line0[p] = line1[p] = make_float2(0.0f, 0.0f);
    __syncthreads();
    if (in) {
      const int count = a.cmax + 4;  // columns -3 .. cmax of rows k, then of rows -k
#pragma unroll 1
      for (int side = 0; side < (k ? 2 : 1); side++) {
        const RowTiles tiles = row_tiles(a, ch, side ? -k : k);
        float2* to = side ? line1 : line0;       // h+ at (c, r)
        float2* mirror = k ? (side ? line0 : line1) : line0;  // h- at (-c, -r)
        for (int i = t; i < count; i += 2 * T) {
          const int c = i - 3;
          const float4 g = cell_at(a, tiles, q, c);
          to[c & (n - 1)] = make_float2(0.5f * g.x, 0.5f * g.y);
          const float2 m = make_float2(0.5f * g.z, -0.5f * g.w);
          if (c > 3) mirror[-c & (n - 1)] = m;
          else near[side * 7 + i] = m;
        }
      }
    }
    __syncthreads();
    for (int i = t; in && i < (k ? 14 : 7); i += 2 * T) {
      const int side = i / 7, c = 3 - i % 7;  // h- of column -c
      float2* to = k ? (side ? line0 : line1) : line0;
      float2 g = to[c & (n - 1)];
      g.x += near[i].x;
      g.y += near[i].y;
      to[c & (n - 1)] = g;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; e++) v[e] = buf[j + e * T];
    __syncthreads();
  } else {
    // Footprints that reach over the grid's edge come back at the other side:
    // rows r and r +- 2N are one line, and so are columns.  First every h+ at its
    // column and the h- that meet no h+ at theirs, then the others (-3 .. 3, and
    // those about the edge); a thread has the same columns, so the same
    // positions, of all rows.
    float2* line0 = smem_f2 + (l & ~1) * S::kStride;
    float2* line1 = line0 + S::kStride;
    const int t = threadIdx.x % (2 * T);
    for (int p = t; p < n; p += 2 * T) line0[p] = line1[p] = make_float2(0.0f, 0.0f);
    __syncthreads();
    auto add = [&](float2* to, int c, float x, float y) {
      const float2 g = to[c & (n - 1)];
      to[c & (n - 1)] = make_float2(fmaf(0.5f, x, g.x), fmaf(0.5f, y, g.y));
    };
    auto lines = [&](auto&& take) {
#pragma unroll 1
      for (int s = 0; in && s < 6; s++) {
        const int side = s & 1, row = (side ? (k ? -k : -N) : k) + (s / 2 - 1) * n;
        const RowTiles tiles = row_tiles(a, ch, row);
        if (tiles.at[0] < 0 && tiles.at[1] < 0) continue;
        // rows 0 and -N are their own mirror images
        take(tiles, side ? line1 : line0, (side != 0) == (k == 0) ? line1 : line0);
      }
    };
    const int edge = n - a.cmax;  // h- of column c >= edge meets an h+
    lines([&](const RowTiles& tiles, float2* to, float2* mirror) {
      for (int c = t - 3; c <= a.cmax; c += 2 * T) {
        const float4 g = cell_at(a, tiles, q, c);
        add(to, c, g.x, g.y);
        if (c > 3 && c < edge) add(mirror, -c, g.z, -g.w);
      }
    });
    __syncthreads();
    lines([&](const RowTiles& tiles, float2*, float2* mirror) {
      for (int i = t; i < 7 + max(0, a.cmax + 1 - edge); i += 2 * T) {
        const int c = i < 7 ? i - 3 : edge + i - 7;
        const float4 g = cell_at(a, tiles, q, c);
        add(mirror, -c, g.z, -g.w);
      }
    });
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 16; e++) v[e] = buf[j + e * T];
    __syncthreads();
  }
  fft16<LG>(v, buf, j, a.tw);
  if (!mine) return;
  // four columns are a sector, and the rows' sectors of these columns lie
  // together: the column pass reads whole lines
  float2* h = a.H + ((size_t)plane * (N / 4) * a.nrow + r - a.rmin) * 4;
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const int col = j + s * T;
    h[(size_t)(col >> 2) * a.nrow * 4 + (col & 3)] = v[kept_output(s)];
  }
}

// Per pixel and channel (blockIdx.y) the factor of the sum that does not
// depend on the image: - fg_scale, beam, GCF and 1/V as the direct engines
// apply them, 0 outside the mask and for a channel without visibilities
// (whose 1/V times its empty sum would be a NaN).  Like the coefficients below it is fixed by
// the problem, made once and laid out column by column ([j][i]), as the
// column pass reads it.
struct FactorArgs {
  int N, normalize, pb;
  float D, pbf, pbcut, fg_scale;
  const float* __restrict__ beam_x;
  const float* __restrict__ beam_y;
  const float* __restrict__ chfreq;
  const int64_t* __restrict__ chnvis;
  const uint8_t* __restrict__ mask;
  const float* __restrict__ gcf;
  float* __restrict__ fac;
};

__global__ void __launch_bounds__(256) k_nu_factors(FactorArgs a) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, MN = (int64_t)a.N * a.N;
  if (q >= MN) return;
  const int c = blockIdx.y;
  const int j = (int)(q / a.N), i = (int)(q - (int64_t)j * a.N);
  const int64_t px = (int64_t)a.N * i + j;
  float f = 0.0f;
  if ((a.mask[px] & kMaskIn) && a.chnvis[c] > 0) {
    f = -(a.fg_scale * attenuation_xy(a.beam_x[j], a.beam_y[i], a.chfreq[c], a.D, a.pbf, a.pbcut,
                                      a.pb));
    if (a.gcf) f *= a.gcf[px];
    if (a.normalize) f /= (float)a.chnvis[c];
  }
  a.fac[c * MN + q] = f;
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
  const int j = (int)(px / N), i = (int)(px - (int64_t)j * N);
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
  int nchan, np, nrow, rmin;  // channels of the group, pairs
  int wterm, alpha;           // alpha: the sum is the alpha plane's
  const float2* __restrict__ H;
  const float2* __restrict__ tw;
  const float* __restrict__ corr;
  const float2* __restrict__ coef;    // [pair][MN]
  const float* __restrict__ fac;      // [channel of the group][MN], or null: 1
  const float* __restrict__ chfreq;   // channel of the group
  float nu_0, fg_scale, threshold;
  const uint8_t* __restrict__ mask;   // pixels written (kMaskIn), or null: all
  const float* __restrict__ img;      // the image's planes (chain rule), or null
  float* __restrict__ out;
  float* part;                        // [block][2][8][kBlock] sums of shared column blocks
  uint32_t* done;                     // [N / kCols] their pieces done
};

// Column FFTs over the covered rows of 2N, the N outputs about the middle
// kept, and the epilogue: every output's real and imaginary part with its
// coefficients, the channel's factor and the chain rule
// (src/functions.cu:3968-4024), summed over pairs and channels in registers.
// kCols adjacent columns per block; kGroups sets of threads take the
// (channel, pair) planes in turn and are added up at the end, so a small
// image's few planes run side by side.
//
// Bound by waits on loads: two blocks an SM is what 64 registers a thread
// allow, and a plane's loads, passes and coefficients follow one another.  16
// planes of 2048^2: 585 us where the traffic takes 86.  With the grid laid out
// row by row, 16 bytes of each for a block's two columns, 695.  Taken back:
// the next plane's rows by cp.async (870), coefficients computed instead of
// read (723), the twiddle factors in shared memory between two sets of
// columns in one block (640).
template <int LG>
struct ColShape {
  static constexpr int kThreads = (1 << LG) / 16;  // per line
  static constexpr int kCols = LG >= 13 ? 1 : (LG == 12 ? 2 : (LG == 11 ? 4 : 2));
  static constexpr int kGroups = LG >= 11 ? 1 : 2;
  // Large sides: the (column block, plane) units in equal runs over two blocks
  // an SM.  1024^2 has 256 column blocks, too few for the 304 places (8
  // channels in two pairs: 187 us with a block each, 178 so); 2048^2 would
  // have 3.4 waves (614 us, 585 so).
  // Blocks whose columns share sectors of the grid take the same run: with one
  // run after the other over single blocks each sector came from HBM twice
  // (2048^2: 1.1 GB, 615 us).
  static constexpr bool kShared = kGroups == 1;
  static constexpr int kTeam = kShared ? 4 / kCols : 1;
  static constexpr int kBlock = kThreads * kCols * kGroups;
  static_assert(!kShared || kBlock == 512, "size of the shared sums");
  // columns are this far apart: 16 / kCols more than a multiple of 16, so the
  // lanes of a half warp, kCols columns wide, fall in distinct banks
  static constexpr int kStride = (span16(1 << LG) + 15) / 16 * 16 + 16 / kCols;
  static constexpr size_t kSmem =
      sizeof(float2) * kGroups * kCols * kStride + sizeof(float) * 8 * kBlock;
};

// (nu / nu_0)^alpha out of line, for the kernels whose length in instructions
// shows: the flat spectra of most images skip it
__device__ __noinline__ float power(float nudiv, float al) {
  return al == 0.0f ? 1.0f : powf(nudiv, al);
}

// The planes of a column block that is shared out between blocks: each leaves
// its sums, and the last to finish adds them up in the planes' order, into
// acc, and goes on with them (true).
template <int kBlock, int kTeam>
__device__ __forceinline__ bool pieces_done(const ColArgs& a, int cblk, int first, int planes,
                                            int cblks, float (&acc)[8]) {
  // a block's piece that starts a column block lies in its second slot
  float* mine = a.part + ((size_t)blockIdx.x * 2 + (first == 0)) * 8 * kBlock + threadIdx.x;
#pragma unroll
  for (int s = 0; s < 8; s++) __stcg(mine + s * kBlock, acc[s]);
  // the runs that hold the column block's first and last unit
  const int64_t total = (int64_t)(cblks / kTeam) * planes;
  const int runs = gridDim.x / kTeam, quad = cblk / kTeam;
  auto holder = [&](int64_t u) {
    int b = (int)(u * runs / total);
    while ((b + 1) * total / runs <= u) b++;
    return b;
  };
  const int b0 = holder((int64_t)quad * planes), b1 = holder((int64_t)(quad + 1) * planes - 1);
  __shared__ int is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    is_last = atomicAdd(a.done + cblk, 1u) == (uint32_t)(b1 - b0);
    if (is_last) a.done[cblk] = 0u;
  }
  __syncthreads();
  const bool mine_to_finish = is_last != 0;
  __syncthreads();  // is_last is read before the next piece sets it
  if (!mine_to_finish) return false;
  __threadfence();
#pragma unroll
  for (int s = 0; s < 8; s++) acc[s] = 0.0f;
  for (int b = b0; b <= b1; b++) {
    const float* p = a.part +
                     ((size_t)(b * kTeam + cblk % kTeam) * 2 + (b == b0)) * 8 * kBlock +
                     threadIdx.x;
#pragma unroll
    for (int s = 0; s < 8; s++) acc[s] += __ldcg(p + s * kBlock);
  }
  return true;
}

template <int LG>
__global__ void __launch_bounds__(ColShape<LG>::kBlock, ColShape<LG>::kBlock == 512 ? 2 : 1)
    k_nu_cols(ColArgs a) {
  using S = ColShape<LG>;
  constexpr int n = 1 << LG, N = n / 2, T = S::kThreads, CB = S::kCols, G = S::kGroups;
  extern __shared__ float2 smem_f2[];
  const int cc = threadIdx.x % CB, j = (threadIdx.x / CB) % T, g = threadIdx.x / (CB * T);
  float2* buf = smem_f2 + (g * CB + cc) * S::kStride;
  constexpr int64_t MN = (int64_t)N * N;
  float* al = reinterpret_cast<float*>(smem_f2 + G * CB * S::kStride) + threadIdx.x;
  const int planes = a.nchan * a.np;
  // this block's units (columns, then planes), see kShared
  int unit = blockIdx.x * planes, end = unit + planes;
  if constexpr (S::kShared) {
    const int64_t total = (int64_t)(N / CB / S::kTeam) * planes;
    const int run = blockIdx.x / S::kTeam, runs = gridDim.x / S::kTeam;
    unit = (int)(run * total / runs);
    end = (int)((run + 1) * total / runs);
  }
#pragma unroll 1
  while (unit < end) {
    const int at = unit / planes, first = unit - at * planes;
    const int cblk = S::kShared ? at * S::kTeam + (int)(blockIdx.x % S::kTeam) : at;
    const int last = min(planes, first + end - unit);
    unit += last - first;
    const int col = cblk * CB + cc;
    // the thread's pixels of the image's alpha plane, kept for all planes; without
    // an image the rounding errors of the planes' sum (a PSF's channels all have
    // one sign)
    bool flat = true;
    if (a.img) {
#pragma unroll
      for (int s = 0; s < 8; s++) {
        const float v = __ldg(a.img + MN + (int64_t)N * (j + s * T) + col);
        al[s * S::kBlock] = v;
        flat = flat && v == 0.0f;
      }
    } else {
#pragma unroll
      for (int s = 0; s < 8; s++) al[s * S::kBlock] = 0.0f;
    }
    // small sides, whose blocks run once through a plane or two: everything the
    // end needs is on its way before the first transform
    constexpr bool kAhead = LG <= 10;
    float old[kAhead ? 8 : 1];
    bool write[kAhead ? 8 : 1];
    if constexpr (kAhead) {
#pragma unroll
      for (int s = 0; s < 8; s++) {
        const int64_t px = (int64_t)N * (j + s * T) + col;
        write[s] = !a.mask || (a.mask[px] & kMaskIn);
        old[s] = a.out[px];
      }
    }
    float acc[8];
#pragma unroll
    for (int s = 0; s < 8; s++) acc[s] = 0.0f;
    for (int p0 = first; p0 < last; p0 += G) {
      const int p = p0 + g;
      const bool in = p < last;
      const int c = p / a.np, q = p - c * a.np;
      float2 v[16];
      {
        // rows below 0 first in memory: row r of the plane at r - rmin
        const float2* h =
            a.H + (((int64_t)p * (N / 4) + (col >> 2)) * a.nrow - a.rmin + j) * 4 + (col & 3);
        const unsigned lo = (unsigned)(j - a.rmin);
#pragma unroll
        for (int e = 0; e < 16; e++) {
          const int o = e < 8 ? e * T : e * T - n;
          v[e] = in && lo + (unsigned)o < (unsigned)a.nrow ? h[4 * o] : make_float2(0.0f, 0.0f);
        }
      }
      const float2* kq = a.coef + q * MN + (int64_t)N * col + j;
      const float* fc = a.fac ? a.fac + c * MN + (int64_t)N * col + j : nullptr;
      float2 kk[kAhead ? 8 : 1];
      float ff[kAhead ? 8 : 1];
      if constexpr (kAhead) {
#pragma unroll
        for (int s = 0; s < 8; s++) {
          kk[s] = in ? __ldg(kq + s * T) : make_float2(0.0f, 0.0f);
          ff[s] = in && fc ? __ldg(fc + s * T) : 1.0f;
        }
      }
      __syncthreads();  // the last line has been read
      fft16<LG>(v, buf, j, a.tw);
      if (!in) continue;
      const float nudiv = a.img ? a.chfreq[c] / a.nu_0 : 1.0f;
      const float lg = a.alpha ? logf(nudiv) : 1.0f;
#pragma unroll
      for (int s = 0; s < 8; s++) {
        const float2 x = v[kept_output(s)];
        float t;
        if (a.wterm) {
          const float2 k = kAhead ? kk[kAhead ? s : 0] : __ldg(kq + s * T);
          t = fmaf(k.x, x.x, k.y * x.y);
        } else {
          t = q == 0 ? x.x * (__ldg(a.corr + j + s * T) * __ldg(a.corr + col)) : 0.0f;
        }
        float f = kAhead ? ff[kAhead ? s : 0] : (fc ? __ldg(fc + s * T) : 1.0f);
        f *= lg;
        if (!flat) {
          const float av = al[s * S::kBlock];
          if constexpr (kAhead) {
            f *= power(nudiv, av);
          } else if (av != 0.0f) {
            f *= powf(nudiv, av);
          }
        }
        if (a.img) {
          acc[s] = fmaf(f, t, acc[s]);
        } else {
          float e = al[s * S::kBlock];
          two_sum(acc[s], e, f * t);
          al[s * S::kBlock] = e;
        }
      }
    }
    if (!a.img) {
#pragma unroll
      for (int s = 0; s < 8; s++) acc[s] += al[s * S::kBlock];
    }
    if constexpr (G > 1) {
      // the groups' sums, in order
      float* part = reinterpret_cast<float*>(smem_f2);
      __syncthreads();
      if (g > 0) {
#pragma unroll
        for (int s = 0; s < 8; s++)
          part[((g - 1) * 8 + s) * T * CB + threadIdx.x % (T * CB)] = acc[s];
      }
      __syncthreads();
      if (g > 0) return;
      for (int o = 0; o < G - 1; o++)
#pragma unroll
        for (int s = 0; s < 8; s++) acc[s] += part[(o * 8 + s) * T * CB + threadIdx.x];
    }
    if constexpr (S::kShared) {
      if (last - first < planes &&
          !pieces_done<S::kBlock, S::kTeam>(a, cblk, first, planes, N / CB, acc))
        continue;
    }
#pragma unroll
    for (int s = 0; s < 8; s++) {
      const int64_t px = (int64_t)N * (j + s * T) + col;
      if (!(kAhead ? write[kAhead ? s : 0] : !a.mask || (a.mask[px] & kMaskIn))) continue;
      float t = acc[s];
      if (a.alpha) {
        const float i0 = a.img[px];
        if (!(i0 > a.threshold)) continue;
        t *= i0 * a.fg_scale;
      }
      a.out[px] = (kAhead ? old[kAhead ? s : 0] : a.out[px]) + t;
    }
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

template <int NP, int W>
gv_status spread_warps(const SpreadArgs& a, cudaStream_t st) {
  const size_t smem = sizeof(float4) * W * (size_t)(NP * kTilePts + NP * 32 + 32 * 5);
  if (smem > 48 * 1024)
    GV_CUDA(cudaFuncSetAttribute(k_nu_spread<NP, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
  k_nu_spread<NP, W><<<a.ntasks, 32 * W, smem, st>>>(a);
  GV_LAUNCH("k_nu_spread");
  return GV_OK;
}

template <int NP>
gv_status spread(const SpreadArgs& a, int warps, cudaStream_t st) {
  return warps == 8 ? spread_warps<NP, 8>(a, st) : spread_warps<NP, 1>(a, st);
}

// blocks of k_nu_cols that share the column blocks out: two an SM
int shared_blocks(const Problem& P) { return 2 * P.num_sms; }

template <int LG>
gv_status transforms(Problem& P, const RowArgs& ra, const ColArgs& ca) {
  using R = RowShape<LG>;
  if (R::kSmem > 48 * 1024)
    GV_CUDA(cudaFuncSetAttribute(k_nu_rows<LG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)R::kSmem));
  k_nu_rows<LG><<<(ra.couples + R::kPairs - 1) / R::kPairs, R::kBlock, R::kSmem, P.stream>>>(ra);
  GV_LAUNCH("k_nu_rows");
  GV_TRY(side_joined(P));  // the priors' gradient is where the sums are added
  using S = ColShape<LG>;
  if (S::kSmem > 48 * 1024)
    GV_CUDA(cudaFuncSetAttribute(k_nu_cols<LG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)S::kSmem));
  int blocks = P.N / S::kCols;
  if (S::kShared)
    blocks = S::kTeam * std::max(1, std::min(blocks / S::kTeam * ca.nchan * ca.np,
                                             shared_blocks(P) / S::kTeam));
  k_nu_cols<LG><<<blocks, S::kBlock, S::kSmem, P.stream>>>(ca);
  GV_LAUNCH("k_nu_cols");
  return GV_OK;
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

// a task's slot, and a channel's grid
size_t slot_bytes(const NuPlan& n) { return sizeof(float4) * kTilePts * n.pairs; }
size_t plane_bytes(const Problem& P) {
  return sizeof(float2) * (size_t)P.nu->pairs * P.nu->nrow * P.N;
}

}  // namespace

void nu_free(Problem& P) {
  if (!P.nu) return;
  NuPlan* n = P.nu;
  cudaFree(n->d_tasks);
  cudaFree(n->d_slot);
  cudaFree(n->d_done);
  cudaFree(n->d_slots);
  cudaFree(n->d_H);
  cudaFree(n->d_twiddle);
  cudaFree(n->d_corr);
  cudaFree(n->d_coef);
  cudaFree(n->d_fac);
  cudaFree(n->d_part);
  delete n;
  P.nu = nullptr;
}

int nu_pairs(const Problem& P) { return P.nu ? P.nu->pairs : 0; }

uint32_t nu_tiles_x(int N) { return (uint32_t)(N / 8 + 1); }

// The plan of P on the host (P.nu stays null where the direct sums are to run):
// keys are the sorted (channel << 32 | tile << 6 | cell in tile) of all
// visibilities, all ones in the low word for those left out.  Its device
// buffers come last of a problem's (nu_build): the direct sums, which need less
// memory, run where there is no room for them, nor for the scratch here.
gv_status nu_plan(Problem& P, const unsigned long long* d_keys, double maxw) {
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
    bool room = true;
    auto take = [&](void* p, size_t bytes) -> gv_status {
      const cudaError_t e = cudaMalloc(static_cast<void**>(p), bytes);
      room = e != cudaErrorMemoryAllocation;
      return e == cudaSuccess ? GV_OK : cuda_fail(e, "nu_plan");
    };
    auto work = [&]() -> gv_status {
      GV_TRY(take(&head, sizeof(int) * V));
      GV_TRY(take(&pos, sizeof(int) * V));
      GV_TRY(take(&tmp, tb));
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
      GV_TRY(take(&dk, sizeof(*dk) * R));
      GV_TRY(take(&ds, sizeof(*ds) * R));
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
    if (!room) {
      cudaGetLastError();
      return GV_OK;
    }
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
  n->cmax = cmax;
  n->rmin = n->wrap ? -N : -rmax;
  n->nrow = n->wrap ? 2 * N : 2 * rmax + 1;
  // ---- tasks ------------------------------------------------------------------
  // A tile's visibilities in pieces of T, a block each.  Few and well filled
  // tiles: the blocks run nearly at once and their longest chain decides, so
  // 8 warps share a piece of 512 (256^2, 104,400 visibilities in 290 tiles).
  // Otherwise one warp a piece, so that none idles in a thin tile, and the dense
  // tiles' pieces do not outlast the rest (2048^2, 8.9 M visibilities in 8
  // channels, an evaluation: 1754 us with pieces of 1024, 1728 of 512, 1735 of
  // 256, which cost more slots: 35 M visibilities 365, 366 and 355 evaluations
  // a second).
  n->warps = R <= (size_t)(16 * P.num_sms) && P.Vgrid >= 64 * (int64_t)R ? 8 : 1;
  const int T = 512;
  std::vector<NuTask>& tasks = n->h_tasks;
  const size_t tiles = (size_t)n->nty * n->ntx;
  std::vector<int>& slot = n->h_slot;
  slot.assign((size_t)C * tiles, -1);
  n->task_off.assign(C + 1, 0);
  for (size_t r = 0; r < R; r++) {
    const uint32_t t = (uint32_t)(rkey[r] & 0x3FFFFFFu);
    const int c = (int)(rkey[r] >> 26);
    const int64_t end_c = P.chans[c].off + P.chans[c].ngrid;
    const int64_t end = (r + 1 < R && (int)(rkey[r + 1] >> 26) == c) ? rstart[r + 1] : end_c;
    const int64_t cnt = end - rstart[r];
    const int parts = (int)((cnt + T - 1) / T);
    const int first = (int)tasks.size();
    for (int k = 0; k < parts; k++) {
      const int64_t b = (int64_t)T * k;
      tasks.push_back({(uint32_t)(rstart[r] + b), (int)std::min<int64_t>(T, cnt - b), first, parts});
    }
    slot[(size_t)c * tiles + (t / NTX - tya) * n->ntx + (t % NTX - txa)] = first;
    n->task_off[c + 1] += parts;
  }
  for (int c = 0; c < C; c++) n->task_off[c + 1] += n->task_off[c];
  // ---- channel groups whose workspace stays bounded ------------------------------
  const size_t slot_b = slot_bytes(*n), h_b = plane_bytes(P);
  n->groups.push_back(0);
  for (int c = 0; c < C;) {
    size_t used = 0;
    const int c0 = c;
    while (c < C) {
      const size_t need = slot_b * (n->task_off[c + 1] - n->task_off[c]) + h_b;
      if (c > c0 && used + need > kWorkspace) break;
      used += need;
      c++;
    }
    n->groups.push_back(c);
    n->max_ch = std::max<size_t>(n->max_ch, c - c0);
    n->max_slots = std::max<size_t>(n->max_slots, n->task_off[c] - n->task_off[c0]);
  }
  return GV_OK;
}

// The plan's device buffers, and the pixels' w-term coefficients and factors:
// once the beam tables (the pixels' offsets), the mask and the channels' tables
// are in place.
gv_status nu_build(Problem& P) {
  if (!P.nu) return GV_OK;
  NuPlan* n = P.nu;
  const int C = (int)P.chans.size(), N = P.N, pairs = n->pairs;
  const std::vector<NuTask>& tasks = n->h_tasks;
  const std::vector<int>& slot = n->h_slot;
  const size_t slot_b = slot_bytes(*n), h_b = plane_bytes(P);
  const size_t fac_b = sizeof(float) * (size_t)N * N;
  const int lg = P.log2n + 1;
  std::vector<float2> tw;
  for (int l = fft16_first(lg); l < lg; l += 4)
    for (int r = 1; r < 16; r++)
      for (int k = 0; k < (1 << l); k++) {
        const double t = 2.0 * kPiD * r * k / (double)(16 << l);
        tw.push_back(make_float2((float)std::cos(t), (float)std::sin(t)));
      }
  const std::vector<float> corr = kernel_correction(N);
  tap_polynomials(n->coef);
  auto upload = [&]() -> cudaError_t {
    cudaError_t e = cudaMalloc(&n->d_tasks, sizeof(NuTask) * tasks.size());
    if (e == cudaSuccess) e = cudaMalloc(&n->d_slot, sizeof(int) * slot.size());
    if (e == cudaSuccess) e = cudaMalloc(&n->d_done, sizeof(uint32_t) * (tasks.size() + N));
    if (e == cudaSuccess) e = cudaMalloc(&n->d_slots, slot_b * n->max_slots);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_H, h_b * n->max_ch);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_twiddle, sizeof(float2) * tw.size());
    if (e == cudaSuccess) e = cudaMalloc(&n->d_corr, sizeof(float) * N);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_coef, sizeof(float2) * (size_t)pairs * N * N);
    if (e == cudaSuccess) e = cudaMalloc(&n->d_fac, fac_b * C);
    if (e == cudaSuccess && N >= 1024)
      e = cudaMalloc(&n->d_part, sizeof(float) * shared_blocks(P) * 2 * 8 * ColShape<11>::kBlock);
    return e;
  };
  const cudaError_t e = upload();
  const size_t large = slot_b * n->max_slots + h_b * n->max_ch + fac_b * C;
  if (e == cudaErrorMemoryAllocation || (e == cudaSuccess && !room_left(large))) {
    // no room for the grids: the direct sums need less
    cudaGetLastError();
    nu_free(P);
    return GV_OK;
  }
  if (e != cudaSuccess) return cuda_fail(e, "nu_build");
  GV_CUDA(cudaMemcpy(n->d_tasks, tasks.data(), sizeof(NuTask) * tasks.size(),
                     cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemcpy(n->d_slot, slot.data(), sizeof(int) * slot.size(), cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemset(n->d_done, 0, sizeof(uint32_t) * (tasks.size() + N)));
  n->tasks = (int)tasks.size();
  GV_CUDA(cudaMemcpy(n->d_twiddle, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemcpy(n->d_corr, corr.data(), sizeof(float) * N, cudaMemcpyHostToDevice));
  n->h_tasks = {};
  n->h_slot = {};
  const int64_t MN = (int64_t)N * N;
  k_nu_coefficients<<<(unsigned)((MN + 255) / 256), 256, 0, P.stream>>>(
      N, pairs, (float)(2.0 * kPiD * n->wmax), P.d_beam_x, P.d_beam_y, n->d_corr, n->d_coef);
  GV_LAUNCH("k_nu_coefficients");
  const FactorArgs fa{N, P.normalize, P.pb, P.D, P.pbf, P.pbcut, P.fg_scale, P.d_beam_x,
                      P.d_beam_y, P.d_chfreq, P.d_chnvis, P.d_mask, P.d_gcf, n->d_fac};
  k_nu_factors<<<dim3((unsigned)((MN + 255) / 256), (unsigned)C), 256, 0, P.stream>>>(fa);
  GV_LAUNCH("k_nu_factors");
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
  sa.done = n.d_done;
  RowArgs ra;
  ra.slots = n.d_slots;
  ra.slot = n.d_slot;
  ra.tw = n.d_twiddle;
  ra.H = n.d_H;
  ra.N = N;
  ra.pairs = np;
  ra.cmax = n.cmax;
  ra.rmin = n.rmin;
  ra.nrow = n.nrow;
  ra.wrap = n.wrap;
  ra.tx0 = n.tx0;
  ra.ntx = n.ntx;
  ra.ty0 = n.ty0;
  ra.nty = n.nty;
  const int64_t MN = (int64_t)P.M * N;
  ColArgs ca;
  ca.part = n.d_part;
  ca.done = n.d_done + n.tasks;
  ca.np = np;
  ca.nrow = n.nrow;
  ca.rmin = n.rmin;
  ca.wterm = mode == 4 ? 0 : 1;
  ca.alpha = mode == 0 && flag_opt % 2 != 0;
  ca.H = n.d_H;
  ca.tw = n.d_twiddle;
  ca.corr = n.d_corr;
  ca.coef = n.d_coef;
  ca.nu_0 = P.nu_0;
  ca.fg_scale = P.fg_scale;
  ca.threshold = P.threshold;
  ca.mask = mode <= 1 ? P.d_mask : nullptr;
  ca.img = mode == 0 ? d_img : nullptr;
  ca.out = d_result + (mode == 0 ? (int64_t)(flag_opt % 2) * MN : 0);
  std::vector<int> one = {only_channel, only_channel + 1};
  const std::vector<int>& groups = only_channel >= 0 ? one : n.groups;
  for (size_t g = 0; g + 1 < groups.size(); g++) {
    const int c0 = groups[g], c1 = groups[g + 1], nch = c1 - c0;
    const int t0 = n.task_off[c0];
    sa.tasks = n.d_tasks + t0;
    sa.ntasks = n.task_off[c1] - t0;
    sa.t0 = t0;
    if (sa.ntasks == 0) continue;
    switch (np) {
      case 1: GV_TRY(spread<1>(sa, n.warps, P.stream)); break;
      case 2: GV_TRY(spread<2>(sa, n.warps, P.stream)); break;
      case 3: GV_TRY(spread<3>(sa, n.warps, P.stream)); break;
      default: GV_TRY(spread<4>(sa, n.warps, P.stream)); break;
    }
    ra.c0 = c0;
    ra.t0 = t0;
    ra.couples = nch * np * (n.wrap ? N : n.nrow / 2 + 1);
    ca.nchan = nch;
    ca.fac = mode <= 1 ? n.d_fac + c0 * MN : nullptr;
    ca.chfreq = P.d_chfreq + c0;
    switch (P.log2n) {
      case 4: GV_TRY(transforms<5>(P, ra, ca)); break;
      case 5: GV_TRY(transforms<6>(P, ra, ca)); break;
      case 6: GV_TRY(transforms<7>(P, ra, ca)); break;
      case 7: GV_TRY(transforms<8>(P, ra, ca)); break;
      case 8: GV_TRY(transforms<9>(P, ra, ca)); break;
      case 9: GV_TRY(transforms<10>(P, ra, ca)); break;
      case 10: GV_TRY(transforms<11>(P, ra, ca)); break;
      case 11: GV_TRY(transforms<12>(P, ra, ca)); break;
      default: GV_TRY(transforms<13>(P, ra, ca)); break;
    }
  }
  return GV_OK;
}

}  // namespace gv
