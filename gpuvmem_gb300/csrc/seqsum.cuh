// The sequential FP32 sum of an array, bit for bit, in parallel.
//
// The reference adds its weights one after another in FP32, so a reduction
// tree would round differently.  But while the running sum s stays in one
// binade, its spacing u is fixed and s + x rounds to s + u round(x / u), the
// increment an integer that does not depend on s, except that an x / u half
// way between two integers goes to the one that makes the sum even.  An
// element is therefore a map from the parity of s / u to an increment, and
// such maps compose associatively.  A block takes a tile of 8192 elements at
// once: without a half in it and within the binade the increments are just
// added; otherwise a scan of the maps gives the sum, or the element at which
// it leaves its binade: that one is added as floats are, and the scan goes on
// from there with the new spacing (some 30 times in a whole array).  Tiles with
// negative, infinite or NaN elements, or sums near the subnormals, are added
// one by one.  Briggs' sums of squares of 16 channels at 1024^2: a chain of
// dependent additions over the half grids 21 ms, this over their occupied
// cells 0.32 ms.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gv {

constexpr int kSeqThreads = 1024, kSeqPer = 8, kSeqTile = kSeqThreads * kSeqPer;

constexpr int kSeqTop = 1 << 24;   // s / u is below this within a binade
constexpr int kSeqFull = 1 << 25;  // increments are held down to this: well past the binade

// increments for an even and an odd sum
struct SeqMap {
  int even, odd;
};
__device__ __forceinline__ SeqMap seq_then(const SeqMap& a, const SeqMap& b) {
  return {min(a.even + ((a.even & 1) ? b.odd : b.even), kSeqFull),
          min(a.odd + ((a.odd & 1) ? b.even : b.odd), kSeqFull)};
}

// the element x / u = y >= 0 as such a map; 2^24 or more leaves any binade
__device__ __forceinline__ SeqMap seq_element(float y) {
  if (!(y < (float)kSeqTop)) return {kSeqTop, kSeqTop};
  const float f = floorf(y), d = y - f;
  const int m = (int)f;
  if (d == 0.5f) return {m + (m & 1), m + 1 - (m & 1)};
  return {m + (d > 0.5f), m + (d > 0.5f)};
}

struct SeqShared {
  float v[kSeqTile + kSeqTile / 32];  // padded: a thread's 8 elements in distinct banks
  SeqMap warp[32];
  int plain[2][32];
  float s;
  int pos;
};
__device__ __forceinline__ int seq_pad(int k) { return k + (k >> 5); }

// s plus load(0), load(1), ... load(n - 1) in order; every thread of a block
// of kSeqThreads calls it and gets the result.
template <class Load>
__device__ float sequential_sum(SeqShared& sh, float s, int64_t n, Load&& load) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  float ahead[kSeqPer];  // the next tile's elements, on their way
#pragma unroll
  for (int k = 0; k < kSeqPer; k++) {
    const int64_t e = tid + k * kSeqThreads;
    ahead[k] = e < n ? load(e) : 0.0f;
  }
  int turn = 0;
  for (int64_t t0 = 0; t0 < n; t0 += kSeqTile) {
    const int cnt = (int)(n - t0 < kSeqTile ? n - t0 : kSeqTile);
    bool odd = false;
    __syncthreads();  // the last tile is done with
#pragma unroll
    for (int k = 0; k < kSeqPer; k++) {
      odd |= !(ahead[k] >= 0.0f && ahead[k] < INFINITY);
      sh.v[seq_pad(tid + k * kSeqThreads)] = ahead[k];
    }
#pragma unroll
    for (int k = 0; k < kSeqPer; k++) {
      const int64_t e = t0 + kSeqTile + tid + k * kSeqThreads;
      ahead[k] = e < n ? load(e) : 0.0f;
    }
    const bool plain = !__syncthreads_or(odd);
    float x[kSeqPer];
#pragma unroll
    for (int k = 0; k < kSeqPer; k++) x[k] = sh.v[seq_pad(tid * kSeqPer + k)];
    int pos = 0;
    while (pos < cnt) {
      if (plain && s == 0.0f) {
        // up to the first element that is not 0
        int first = cnt;
#pragma unroll
        for (int k = kSeqPer - 1; k >= 0; k--)
          if (x[k] != 0.0f && tid * kSeqPer + k >= pos && tid * kSeqPer + k < cnt)
            first = tid * kSeqPer + k;
        if (tid == 0) sh.pos = cnt;
        __syncthreads();
        if (first < cnt) atomicMin(&sh.pos, first);
        __syncthreads();
        pos = sh.pos;
        __syncthreads();
        if (pos < cnt) s = __fadd_rn(s, sh.v[seq_pad(pos++)]);
        continue;
      }
      if (!plain || !(s >= 1e-30f && s < 1e38f)) {
        if (tid == 0) {
          for (int k = pos; k < cnt; k++) s = __fadd_rn(s, sh.v[seq_pad(k)]);
          sh.s = s;
        }
        __syncthreads();
        s = sh.s;
        pos = cnt;
        continue;
      }
      int ex;
      frexpf(s, &ex);                                 // s in [2^(ex-1), 2^ex)
      const float u = ldexpf(1.0f, ex - 24), inv = ldexpf(1.0f, 24 - ex);
      const int S = (int)(s * inv), top = kSeqTop;
      if (pos == 0) {
        // no halves and no step out of the binade: the increments' plain sum
        int sum = 0;
        bool half = false;
#pragma unroll
        for (int k = 0; k < kSeqPer; k++) {
          const SeqMap m = seq_element(x[k] * inv);  // elements past cnt are 0
          sum += m.even;
          half |= m.even != m.odd;
        }
        const int w = __reduce_add_sync(0xffffffffu, min(sum, kSeqFull));
        turn ^= 1;
        if (lane == 0) sh.plain[turn][wid] = min(w, kSeqFull);
        if (!__syncthreads_or(half)) {
          const int total = __reduce_add_sync(0xffffffffu, sh.plain[turn][lane]);
          if (total < top - S) {
            s = (float)(S + total) * u;
            pos = cnt;
            continue;
          }
        }
      }
      SeqMap mine{0, 0};
#pragma unroll
      for (int k = 0; k < kSeqPer; k++) {
        const int e = tid * kSeqPer + k;
        if (e >= pos && e < cnt) mine = seq_then(mine, seq_element(x[k] * inv));
      }
      // inclusive scan over the block
      SeqMap inc = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const SeqMap p{__shfl_up_sync(0xffffffffu, inc.even, o),
                       __shfl_up_sync(0xffffffffu, inc.odd, o)};
        if (lane >= o) inc = seq_then(p, inc);
      }
      if (lane == 31) sh.warp[wid] = inc;
      __syncthreads();
      if (wid == 0) {
        SeqMap w = sh.warp[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const SeqMap p{__shfl_up_sync(0xffffffffu, w.even, o),
                         __shfl_up_sync(0xffffffffu, w.odd, o)};
          if (lane >= o) w = seq_then(p, w);
        }
        sh.warp[lane] = w;
      }
      __syncthreads();
      const bool odd_s = S & 1;
      const int total = odd_s ? sh.warp[31].odd : sh.warp[31].even;
      if (S + total < top) {
        s = (float)(S + total) * u;
        pos = cnt;
        __syncthreads();  // sh.warp is written again
        continue;
      }
      // the sum before this thread's elements
      SeqMap before{__shfl_up_sync(0xffffffffu, inc.even, 1),
                    __shfl_up_sync(0xffffffffu, inc.odd, 1)};
      if (lane == 0) before = {0, 0};
      if (wid > 0) before = seq_then(sh.warp[wid - 1], before);
      int at = S + (odd_s ? before.odd : before.even);
      if (at < top) {
#pragma unroll
        for (int k = 0; k < kSeqPer; k++) {
          const int e = tid * kSeqPer + k;
          if (e < pos || e >= cnt || at >= top) continue;
          const SeqMap m = seq_element(x[k] * inv);
          const int next = at + ((at & 1) ? m.odd : m.even);
          if (next >= top) {  // the one element at which the sum leaves the binade
            sh.s = __fadd_rn((float)at * u, x[k]);
            sh.pos = e + 1;
          }
          at = next;
        }
      }
      __syncthreads();
      s = sh.s;
      pos = sh.pos;
      __syncthreads();
    }
  }
  return s;
}

}  // namespace gv
