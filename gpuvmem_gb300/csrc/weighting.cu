// Visibility weighting schemes on the GPU: NaturalWeightingScheme::apply
// (src/naturalweightingscheme.cu:9-52), UniformWeightingScheme::apply
// (src/uniformweightingscheme.cu:9-102) and BriggsWeightingScheme::apply
// (src/briggsweightingscheme.cu:30-190), one field and one correlation,
// without a uv taper.
//
// The reference grids the weights in FP32 with an OpenMP critical section
// per visibility, so its result depends on the thread schedule; with one
// thread it is a sequential FP32 sum per grid cell in visibility order.
// This version reproduces that one-thread result bit for bit without a
// critical section: the visibilities of all channels are sorted by (cell,
// channel) with a stable radix sort, and one thread per occupied cell adds
// that cell's weights in visibility order, channel after channel (Briggs'
// cumulative first pass).  The scalar sums that feed Briggs' f^2, of the
// weights and of the squares of the half grid after each channel, keep the
// reference's sequential FP32 order (seqsum.cuh); cells without a weight add
// nothing, so only occupied ones enter.  Data too large for one sort (or for
// the table of sums per channel and cell) go channel by channel.

#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "gv_internal.cuh"
#include "seqsum.cuh"

namespace gv {
namespace {

constexpr uint32_t kNoCell = 0xFFFFFFFFu;
// half a side at most: grids end at 4096, as images do
constexpr int kMaxHalf = 2048;
// bounds of the one-sort path: visibilities, and floats of the table of sums
constexpr int64_t kOneSort = int64_t(1) << 28, kTable = int64_t(1) << 30;

// cell of every visibility (src/briggsweightingscheme.cu:74-88): float
// wavelength, u < 0 flipped, truncation of u / |du| + N/2 + 0.5
__global__ void k_weight_cells(int64_t n, const double* __restrict__ uvw, float freq, double adu,
                               double adv, int M, int N, uint32_t* __restrict__ key,
                               uint32_t* __restrict__ idx) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const float lambda = kLightSpeed / freq;
  double u = uvw[3 * k] / lambda, v = uvw[3 * k + 1] / lambda;
  if (u < 0.0) {
    u *= -1.0;
    v *= -1.0;
  }
  const int x = (int)(u / adu + (double)(N / 2) + 0.5);
  const int y = (int)(v / adv + (double)(M / 2) + 0.5);
  key[k] = (x >= 0 && y >= 0 && x < N && y < M) ? (uint32_t)(N * y + x) : kNoCell;
  idx[k] = (uint32_t)k;
}

// one thread per run of equal keys: grid[cell] += w of the run, in order
__global__ void k_cell_runs(int64_t n, const uint32_t* __restrict__ key,
                            const uint32_t* __restrict__ idx, const float* __restrict__ w,
                            float* __restrict__ grid) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t c = key[k];
  if (c == kNoCell || (k > 0 && key[k - 1] == c)) return;
  float s = grid[c];
  for (int64_t j = k; j < n && key[j] == c; j++) s += w[idx[j]];
  grid[c] = s;
}

// sum over rows m and columns N/2..N-1 of grid^2, in that order, added to *acc
__global__ void __launch_bounds__(kSeqThreads) k_half_sumsq(int M, int N,
                                                            const float* __restrict__ grid,
                                                            float* __restrict__ acc) {
  __shared__ SeqShared sh;
  const int x0 = N / 2, half = N - N / 2;
  const float s = sequential_sum(sh, *acc, (int64_t)M * half, [=](int64_t k) {
    const int64_t m = k / half;
    const float g = grid[(int64_t)N * m + x0 + (k - m * half)];
    return g * g;
  });
  __syncthreads();
  if (threadIdx.x == 0) *acc = s;
}

// ---- all channels in one sort ------------------------------------------------
// (cell, channel) of every visibility; the visibilities of channel c are
// off[c] .. off[c + 1] - 1
__global__ void k_cell_keys(int C, const int64_t* __restrict__ off, const float* __restrict__ freq,
                            const double* __restrict__ uvw, double adu, double adv, int M, int N,
                            uint32_t* __restrict__ key, uint32_t* __restrict__ idx) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= off[C]) return;
  int c = 0, hi = C;  // off[c] <= k < off[hi]
  while (hi - c > 1) {
    const int m = (c + hi) >> 1;
    if (off[m] <= k) c = m;
    else hi = m;
  }
  const float lambda = kLightSpeed / freq[c];
  double u = uvw[3 * k] / lambda, v = uvw[3 * k + 1] / lambda;
  if (u < 0.0) {
    u *= -1.0;
    v *= -1.0;
  }
  const int x = (int)(u / adu + (double)(N / 2) + 0.5);
  const int y = (int)(v / adv + (double)(M / 2) + 0.5);
  key[k] = (x >= 0 && y >= 0 && x < N && y < M) ? (uint32_t)(N * y + x) * (uint32_t)C + c : kNoCell;
  idx[k] = (uint32_t)k;
}

// weights in sorted order; first visibilities of the cells of the half grid
__global__ void k_sorted(int64_t n, int C, int N, const uint32_t* __restrict__ key,
                         const uint32_t* __restrict__ idx, const float* __restrict__ w,
                         float* __restrict__ ws, int* __restrict__ head) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  ws[k] = w[idx[k]];
  const uint32_t q = key[k], cell = q / C;
  head[k] = q != kNoCell && (int)(cell % N) >= N / 2 && (k == 0 || key[k - 1] / C != cell);
}

// s plus the weights from j on whose key is q, in order; j moves past them.
// Eight at a time: their loads are in flight together.
__device__ __forceinline__ float run_sum(float s, int64_t& j, int64_t n, uint32_t q,
                                         const uint32_t* __restrict__ key,
                                         const float* __restrict__ ws) {
  for (;;) {
    uint32_t k[8];
    float x[8];
#pragma unroll
    for (int t = 0; t < 8; t++) {
      const bool in = j + t < n;
      k[t] = in ? key[j + t] : ~q;
      x[t] = in ? ws[j + t] : 0.0f;
    }
    int t = 0;
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (t == u && k[u] == q) {
        s = __fadd_rn(s, x[u]);
        t = u + 1;
      }
    j += t;
    if (t < 8) return s;
  }
}

// one thread per cell of the half grid: its cumulative sum after every channel
// (G[channel][cell], the cells in grid order)
__global__ void k_cumulative(int64_t n, int C, const uint32_t* __restrict__ key,
                             const float* __restrict__ ws, const int* __restrict__ head,
                             const int* __restrict__ pos, int64_t cells, float* __restrict__ G) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n || !head[k]) return;
  const uint32_t first = key[k] - key[k] % C;
  float s = 0.0f;
  int64_t j = k;
  for (int c = 0; c < C; c++) {
    s = run_sum(s, j, n, first + c, key, ws);
    G[c * cells + pos[k]] = s;
  }
}

// first visibilities of the (cell, channel) runs
__global__ void k_run_heads(int64_t n, const uint32_t* __restrict__ key, int* __restrict__ head) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) head[k] = k == 0 || key[k - 1] != key[k];
}

// one thread per run: the channel's own sum of the cell
__global__ void k_run_sums(int64_t n, const uint32_t* __restrict__ key,
                           const float* __restrict__ ws, const int* __restrict__ head,
                           const int* __restrict__ run, float* __restrict__ sum) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n || !head[k] || key[k] == kNoCell) return;
  int64_t e = k;
  sum[run[k]] = run_sum(0.0f, e, n, key[k], key, ws);
}

__global__ void k_reweight(int64_t n, int briggs, float f2, const uint32_t* __restrict__ key,
                           const uint32_t* __restrict__ idx, const float* __restrict__ ws,
                           const int* __restrict__ head, const int* __restrict__ run,
                           const float* __restrict__ sum, float* __restrict__ out) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  float r = 0.0f;
  if (key[k] != kNoCell) {
    const float s = sum[run[k] + head[k] - 1];
    r = briggs ? (float)((double)ws[k] / (1.0 + (double)(s * f2))) : ws[k] / s;
  }
  out[idx[k]] = r;
}

// sums[c] = the channel's weights, sums[C] = the squares of G, each in order
__global__ void __launch_bounds__(kSeqThreads) k_scalar_sums(int C, const int64_t* __restrict__ off,
                                                             const float* __restrict__ w,
                                                             int64_t ng, const float* __restrict__ G,
                                                             float* __restrict__ sums) {
  __shared__ SeqShared sh;
  const int c = blockIdx.x;
  float s;
  if (c < C) {
    const float* wc = w + off[c];
    s = sequential_sum(sh, 0.0f, off[c + 1] - off[c], [wc](int64_t k) { return wc[k]; });
  } else {
    s = sequential_sum(sh, 0.0f, ng, [G](int64_t k) { return G[k] * G[k]; });
  }
  if (threadIdx.x == 0) sums[c] = s;
}

__global__ void k_apply_uniform(int64_t n, const uint32_t* __restrict__ cell,
                                const float* __restrict__ grid, float* __restrict__ w) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t c = cell[k];
  w[k] = c != kNoCell ? w[k] / grid[c] : 0.0f;
}

__global__ void k_apply_briggs(int64_t n, const uint32_t* __restrict__ cell,
                               const float* __restrict__ grid, float f2, float* __restrict__ w) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t c = cell[k];
  w[k] = c != kNoCell ? (float)((double)w[k] / (1.0 + (double)(grid[c] * f2))) : 0.0f;
}

struct Buffers {
  double* uvw = nullptr;
  float* w = nullptr;
  uint32_t *key = nullptr, *idx = nullptr, *skey = nullptr, *sidx = nullptr;
  float* grid = nullptr;
  float* acc = nullptr;
  void* tmp = nullptr;
  size_t tmp_bytes = 0;
  ~Buffers() {
    cudaFree(uvw);
    cudaFree(w);
    cudaFree(key);
    cudaFree(idx);
    cudaFree(skey);
    cudaFree(sidx);
    cudaFree(grid);
    cudaFree(acc);
    cudaFree(tmp);
  }
};

// Copies of the channels' arrays that lie one after another on the host as one
// array go as one copy (a user's channels are slices of one); one by one where
// they only happen to be neighbours, each pinned by itself, which a copy may not
// span.
template <class T, class F>
cudaError_t copy_channels(int C, const int64_t* off, int width, cudaStream_t st, T* dev, F&& host,
                          cudaMemcpyKind kind) {
  auto copy = [&](int c, int e) {  // channels c .. e - 1
    auto* h = host(c);
    T* d = dev + off[c] * width;
    const size_t bytes = sizeof(T) * (size_t)(off[e] - off[c]) * width;
    return kind == cudaMemcpyHostToDevice ? cudaMemcpyAsync(d, (const void*)h, bytes, kind, st)
                                          : cudaMemcpyAsync((void*)h, d, bytes, kind, st);
  };
  for (int c = 0; c < C;) {
    int e = c + 1;
    if (off[e] > off[c]) {
      auto* h = host(c);
      while (e < C && (off[e + 1] == off[e] || host(e) == h + (off[e] - off[c]) * width)) e++;
      cudaError_t err = copy(c, e);
      if (err == cudaErrorInvalidValue && e > c + 1) {
        cudaGetLastError();
        err = cudaSuccess;
        for (int k = c; k < e && err == cudaSuccess; k++)
          if (off[k + 1] > off[k]) err = copy(k, k + 1);
      }
      if (err != cudaSuccess) return err;
    }
    c = e;
  }
  return cudaSuccess;
}

// Uniform and Briggs weights of all channels from one sort; *done is false
// (and nothing written) where the data are beyond its bounds or do not fit.
gv_status weights_in_one_sort(bool briggs, float robust, int M, int N, double adu, double adv,
                              int C, const gv_channel_desc* ch, float* const* out, cudaStream_t st,
                              bool* done) {
  *done = false;
  std::vector<int64_t> off(C + 1, 0);
  std::vector<float> freq(C);
  for (int c = 0; c < C; c++) {
    off[c + 1] = off[c] + ch[c].nvis;
    freq[c] = ch[c].freq_hz;
  }
  const int64_t V = off[C], MN = (int64_t)M * N;
  if (V == 0) {
    *done = true;
    return GV_OK;
  }
  const int64_t table = briggs ? (int64_t)C * std::min<int64_t>(V, MN / 2 + M) : 1;
  if (V > kOneSort || MN * C >= (int64_t)kNoCell || table > kTable) return GV_OK;
  int bits = 0;
  while (bits < 32 && ((MN * C) >> bits) != 0) bits++;  // all ones stay the largest key
  const size_t tmp_b = std::max(radix_sort_scratch<uint32_t, uint32_t>(V), scan_scratch(V));
  Arena a;
  double* uvw = nullptr;
  float *w = nullptr, *ws = nullptr, *G = nullptr, *sums = nullptr, *d_freq = nullptr;
  uint32_t *key = nullptr, *idx = nullptr, *skey = nullptr, *sidx = nullptr;
  int *head = nullptr, *pos = nullptr;
  int64_t* d_off = nullptr;
  void* tmp = nullptr;
  for (int pass = 0; pass < 2; pass++) {
    a.used = 0;
    uvw = a.take<double>(3 * V);
    w = a.take<float>(V);
    ws = a.take<float>(V);
    key = a.take<uint32_t>(V);
    idx = a.take<uint32_t>(V);
    skey = a.take<uint32_t>(V);
    sidx = a.take<uint32_t>(V);
    head = a.take<int>(V);
    pos = a.take<int>(V);
    G = a.take<float>(table);
    sums = a.take<float>(C + 1);
    d_freq = a.take<float>(C);
    d_off = a.take<int64_t>(C + 1);
    tmp = a.take<unsigned char>((int64_t)tmp_b);
    if (pass == 0 && cudaMalloc(&a.p, a.used) != cudaSuccess) {
      cudaGetLastError();
      return GV_OK;
    }
  }
  GV_CUDA(copy_channels(C, off.data(), 3, st, uvw, [&](int c) { return ch[c].uvw; },
                        cudaMemcpyHostToDevice));
  GV_CUDA(copy_channels(C, off.data(), 1, st, w, [&](int c) { return ch[c].weight; },
                        cudaMemcpyHostToDevice));
  GV_CUDA(cudaMemcpyAsync(d_off, off.data(), sizeof(int64_t) * (C + 1), cudaMemcpyHostToDevice, st));
  GV_CUDA(cudaMemcpyAsync(d_freq, freq.data(), sizeof(float) * C, cudaMemcpyHostToDevice, st));
  const unsigned gb = (unsigned)((V + 255) / 256);
  k_cell_keys<<<gb, 256, 0, st>>>(C, d_off, d_freq, uvw, adu, adv, M, N, key, idx);
  GV_LAUNCH("k_cell_keys");
  GV_TRY((radix_sort_pairs<uint32_t, uint32_t>(tmp, tmp_b, key, skey, idx, sidx, V, 0, bits, st)));
  k_sorted<<<gb, 256, 0, st>>>(V, C, N, skey, sidx, w, ws, head);
  GV_LAUNCH("k_sorted");
  float f2 = 0.0f;
  if (briggs) {
    GV_TRY(exclusive_scan<int>(tmp, tmp_b, head, pos, V, st));
    int last[2] = {0, 0};
    GV_CUDA(cudaMemcpyAsync(&last[0], head + V - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    GV_CUDA(cudaMemcpyAsync(&last[1], pos + V - 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    GV_CUDA(cudaStreamSynchronize(st));
    const int64_t cells = (int64_t)last[0] + last[1];
    k_cumulative<<<gb, 256, 0, st>>>(V, C, skey, ws, head, pos, cells, G);
    GV_LAUNCH("k_cumulative");
    k_scalar_sums<<<C + 1, kSeqThreads, 0, st>>>(C, d_off, w, cells * C, G, sums);
    GV_LAUNCH("k_scalar_sums");
    std::vector<float> h(C + 1);
    GV_CUDA(cudaMemcpyAsync(h.data(), sums, sizeof(float) * (C + 1), cudaMemcpyDeviceToHost, st));
    GV_CUDA(cudaStreamSynchronize(st));
    float sum_orig = 0.0f;
    for (int c = 0; c < C; c++) sum_orig += h[c];
    const float average = h[C] / sum_orig;
    const float r = 5.0f * powf(10.0f, -robust);
    f2 = r * r / average;
  }
  k_run_heads<<<gb, 256, 0, st>>>(V, skey, head);
  GV_LAUNCH("k_run_heads");
  GV_TRY(exclusive_scan<int>(tmp, tmp_b, head, pos, V, st));
  float* own = reinterpret_cast<float*>(key);  // the unsorted keys are done with
  k_run_sums<<<gb, 256, 0, st>>>(V, skey, ws, head, pos, own);
  GV_LAUNCH("k_run_sums");
  k_reweight<<<gb, 256, 0, st>>>(V, briggs ? 1 : 0, f2, skey, sidx, ws, head, pos, own, w);
  GV_LAUNCH("k_reweight");
  GV_CUDA(copy_channels(C, off.data(), 1, st, w, [&](int c) { return out[c]; },
                        cudaMemcpyDeviceToHost));
  GV_CUDA(cudaStreamSynchronize(st));
  *done = true;
  return GV_OK;
}

}  // namespace
}  // namespace gv

extern "C" gv_status gv_apply_weighting(int32_t scheme, float robust, int32_t M, int32_t N,
                                        double deltax_deg, double deltay_deg, int32_t nchannels,
                                        const gv_channel_desc* ch, float* const* weights_out,
                                        void* stream) {
  using namespace gv;
  if (scheme < GV_WEIGHT_NATURAL || scheme > GV_WEIGHT_BRIGGS || M < 2 || N < 2 ||
      N - N / 2 > kMaxHalf ||
      nchannels < 1 || !ch || !weights_out || deltax_deg == 0.0 || deltay_deg == 0.0) {
    set_error("invalid weighting arguments");
    return GV_ERR_INVALID;
  }
  for (int c = 0; c < nchannels; c++)
    if (ch[c].nvis < 0 || (ch[c].nvis > 0 && (!ch[c].uvw || !ch[c].weight || !weights_out[c])) ||
        ch[c].nvis >= (int64_t)kNoCell) {
      set_error("invalid channel in weighting");
      return GV_ERR_INVALID;
    }
  // deltau = 1 / (M * deltax), deltax = RPDEG_D * DELTAX (src/mfs.cu:531-534)
  const double deltax = kRpDegD * deltax_deg, deltay = kRpDegD * deltay_deg;
  const double adu = std::fabs(1.0 / ((double)M * deltax));
  const double adv = std::fabs(1.0 / ((double)N * deltay));
  if (scheme == GV_WEIGHT_NATURAL) {
    for (int c = 0; c < nchannels; c++)
      if (weights_out[c] != ch[c].weight)
        std::copy(ch[c].weight, ch[c].weight + ch[c].nvis, weights_out[c]);
    return GV_OK;
  }
  cudaStream_t st = (cudaStream_t)stream;
  bool done = false;
  GV_TRY(weights_in_one_sort(scheme == GV_WEIGHT_BRIGGS, robust, M, N, adu, adv, nchannels, ch,
                             weights_out, st, &done));
  if (done) return GV_OK;
  int64_t vmax = 1;
  for (int c = 0; c < nchannels; c++) vmax = std::max<int64_t>(vmax, ch[c].nvis);
  const int64_t MN = (int64_t)M * N;
  Buffers b;
  GV_CUDA(cudaMalloc(&b.uvw, sizeof(double) * 3 * vmax));
  GV_CUDA(cudaMalloc(&b.w, sizeof(float) * vmax));
  GV_CUDA(cudaMalloc(&b.key, sizeof(uint32_t) * vmax));
  GV_CUDA(cudaMalloc(&b.idx, sizeof(uint32_t) * vmax));
  GV_CUDA(cudaMalloc(&b.skey, sizeof(uint32_t) * vmax));
  GV_CUDA(cudaMalloc(&b.sidx, sizeof(uint32_t) * vmax));
  GV_CUDA(cudaMalloc(&b.grid, sizeof(float) * MN));
  GV_CUDA(cudaMalloc(&b.acc, sizeof(float)));
  b.tmp_bytes = radix_sort_scratch<uint32_t, uint32_t>(vmax);
  GV_CUDA(cudaMalloc(&b.tmp, b.tmp_bytes));
  // grid one channel's weights into b.grid (added to what it holds)
  auto grid_channel = [&](int c) -> gv_status {
    const int64_t n = ch[c].nvis;
    if (n == 0) return GV_OK;
    GV_CUDA(cudaMemcpyAsync(b.uvw, ch[c].uvw, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, st));
    GV_CUDA(cudaMemcpyAsync(b.w, ch[c].weight, sizeof(float) * n, cudaMemcpyHostToDevice, st));
    const unsigned gb = (unsigned)((n + 255) / 256);
    k_weight_cells<<<gb, 256, 0, st>>>(n, b.uvw, ch[c].freq_hz, adu, adv, M, N, b.key, b.idx);
    GV_LAUNCH("k_weight_cells");
    GV_TRY((radix_sort_pairs<uint32_t, uint32_t>(b.tmp, b.tmp_bytes, b.key, b.skey, b.idx,
                                                  b.sidx, n, 0, 32, st)));
    k_cell_runs<<<gb, 256, 0, st>>>(n, b.skey, b.sidx, b.w, b.grid);
    GV_LAUNCH("k_cell_runs");
    return GV_OK;
  };
  float f2 = 0.0f;
  if (scheme == GV_WEIGHT_BRIGGS) {
    // sum of the original weights (std::accumulate per channel, FP32)
    float sum_orig = 0.0f;
    for (int c = 0; c < nchannels; c++)
      sum_orig += std::accumulate(ch[c].weight, ch[c].weight + ch[c].nvis, 0.0f);
    GV_CUDA(cudaMemsetAsync(b.grid, 0, sizeof(float) * MN, st));
    GV_CUDA(cudaMemsetAsync(b.acc, 0, sizeof(float), st));
    for (int c = 0; c < nchannels; c++) {
      GV_TRY(grid_channel(c));  // cumulative over channels, as the reference
      k_half_sumsq<<<1, kSeqThreads, 0, st>>>(M, N, b.grid, b.acc);
      GV_LAUNCH("k_half_sumsq");
    }
    float sum_sq = 0.0f;
    GV_CUDA(cudaMemcpyAsync(&sum_sq, b.acc, sizeof(float), cudaMemcpyDeviceToHost, st));
    GV_CUDA(cudaStreamSynchronize(st));
    const float average = sum_sq / sum_orig;
    const float r = 5.0f * powf(10.0f, -robust);
    f2 = r * r / average;
  }
  for (int c = 0; c < nchannels; c++) {
    const int64_t n = ch[c].nvis;
    if (n == 0) continue;
    GV_CUDA(cudaMemsetAsync(b.grid, 0, sizeof(float) * MN, st));
    GV_TRY(grid_channel(c));
    const unsigned gb = (unsigned)((n + 255) / 256);
    if (scheme == GV_WEIGHT_UNIFORM)
      k_apply_uniform<<<gb, 256, 0, st>>>(n, b.key, b.grid, b.w);
    else
      k_apply_briggs<<<gb, 256, 0, st>>>(n, b.key, b.grid, f2, b.w);
    GV_LAUNCH("k_apply_weights");
    GV_CUDA(cudaMemcpyAsync(weights_out[c], b.w, sizeof(float) * n, cudaMemcpyDeviceToHost, st));
    GV_CUDA(cudaStreamSynchronize(st));
  }
  return GV_OK;
}
