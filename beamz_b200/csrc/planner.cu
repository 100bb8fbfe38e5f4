// On-device planning: monitor gather plans packed per point (nonzero weights
// first, offsets remapped to the device layout), the voxel-id histogram
// behind the codebook's compact material indices, and 2D gather slots sorted by
// the cell that they read.  beamz does the first two on the host
// (beamz/simulation/cuda/runtime.py:530-618, compile.py:146-187).

#include "kernels.cuh"

namespace fdtd {

namespace {

constexpr int kPackThreads = 256;
constexpr int kMaxSlots = 32;

__device__ __forceinline__ int remap_offset(int flat, const GatherPackDev& g) {
  const int64_t n = static_cast<int64_t>(g.dz) * g.dy * g.dx;
  if (flat < 0 || flat >= n) return -1;
  const int i = flat % g.dx;
  const int r = flat / g.dx;
  const int j = r % g.dy, k = r / g.dy;
  return static_cast<int>(k * g.plane + j * g.row + i);
}

__global__ void __launch_bounds__(kPackThreads) gather_pack_kernel(GatherPackDev g) {
  const int p = blockIdx.x * kPackThreads + threadIdx.x;
  if (p >= g.points) return;
  const int* idx = g.idx_in + static_cast<int64_t>(p) * g.slots_in;
  const float* w = g.w_in + static_cast<int64_t>(p) * g.slots_in;
  int n = 0;
  for (int pass = 0; pass < 2; ++pass) {  // nonzero weights, then zero weights
    for (int s = 0; s < g.slots_in; ++s) {
      const float ws = w[s];
      if ((ws != 0.0f) != (pass == 0)) continue;
      if (n < g.rows) {  // rows past the output's K hold only zero weights (the caller sizes K)
        g.idx_out[static_cast<int64_t>(n) * g.pmax + p] = remap_offset(idx[s], g);
        g.w_out[static_cast<int64_t>(n) * g.pmax + p] = ws;
      }
      ++n;
    }
  }
}

__global__ void __launch_bounds__(kPackThreads) voxel_histogram_kernel(const uint8_t* v, int64_t n, int* counts) {
  __shared__ int h[256];
  for (int b = threadIdx.x; b < 256; b += kPackThreads) h[b] = 0;
  __syncthreads();
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * kPackThreads + threadIdx.x; e < n;
       e += static_cast<int64_t>(gridDim.x) * kPackThreads)
    atomicAdd(&h[v[e]], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < 256; b += kPackThreads)
    if (h[b]) atomicAdd(&counts[b], h[b]);
}

// The block (component, row, 16 columns) of slot t of the sorted ones, the last
// block + 1 for a slot that is not sampled; *at: its offset in the plan.
__device__ __forceinline__ int slot_block(const SlotSortDev& d, int t, int* at) {
  const int p = t % d.P, r = t / d.P, k = r % d.K, ma = r / d.K, m = ma / d.n, a = ma - m * d.n;
  const int c = a == 0 ? d.comp[0] : (a == 1 ? d.comp[1] : d.comp[2]);
  const int width = a == 0 ? d.width[0] : (a == 1 ? d.width[1] : d.width[2]);
  const int height = a == 0 ? d.height[0] : (a == 1 ? d.height[1] : d.height[2]);
  const int point = (m * d.C + c) * d.K * d.P + p;
  *at = point + k * d.P;
  const int none = d.n * d.rows * d.blocks;
  if (d.masks != nullptr && d.masks[m * d.C + c] == 0.0f) return none;
  for (int s = 0; s <= k; ++s)  // a zero weight ends a point's gather
    if (d.w[point + s * d.P] == 0.0f) return none;
  const int idx = d.idx[*at];
  if (idx < 0 || idx / width >= height) return none;
  const int y = idx / width;
  return (a * d.rows + y) * d.blocks + (idx - y * width) / kSlotBlock;
}

// Counts per block, then (Fill, after the scan) the slots: `first` holds the end of
// each block, is counted down, and ends as its start.
template <bool Fill>
__global__ void __launch_bounds__(kPackThreads) slot_count_kernel(SlotSortDev d, int total) {
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kPackThreads + threadIdx.x; t < total;
       t += static_cast<int64_t>(gridDim.x) * kPackThreads) {
    int at;
    const int b = slot_block(d, static_cast<int>(t), &at);
    if constexpr (Fill) {
      const int to = atomicSub(&d.first[b], 1) - 1;
      if (to >= 0 && to < total) d.order[to] = at;
    } else {
      atomicAdd(&d.first[b], 1);
    }
  }
}

constexpr int kScanThreads = 1024, kScanEach = 8;

// In-place inclusive sums by one block, 8192 entries at a time (190 000 of them at
// 1000 x 1000 cells; a program's compilation has this once).
__global__ void __launch_bounds__(kScanThreads) slot_scan_kernel(int* v, int n) {
  __shared__ int sums[kScanThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int carry = 0;
  for (int base = 0; base < n; base += kScanThreads * kScanEach) {
    const int at = base + tid * kScanEach;
    int x[kScanEach];
#pragma unroll
    for (int q = 0; q < kScanEach; ++q) x[q] = at + q < n ? v[at + q] : 0;
#pragma unroll
    for (int q = 1; q < kScanEach; ++q) x[q] += x[q - 1];
    int s = x[kScanEach - 1];  // inclusive over the warp, then over the block
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += u;
    }
    if (lane == 31) sums[warp] = s;
    __syncthreads();
    int before = carry, all = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) {
      if (w < warp) before += sums[w];
      all += sums[w];
    }
    before += s - x[kScanEach - 1];
#pragma unroll
    for (int q = 0; q < kScanEach; ++q)
      if (at + q < n) v[at + q] = before + x[q];
    carry += all;
    __syncthreads();  // the sums, before the next round writes them
  }
}

}  // namespace

cudaError_t launch_slot_order(cudaStream_t s, const SlotSortDev& d) {
  const int64_t total = static_cast<int64_t>(d.M) * d.n * d.K * d.P;
  const int64_t bins = static_cast<int64_t>(d.n) * d.rows * d.blocks + 1;
  cudaError_t err = cudaMemsetAsync(d.first, 0, bins * sizeof(int), s);
  if (err != cudaSuccess || total <= 0) return err;
  const int64_t want = (total + kPackThreads - 1) / kPackThreads;
  const int blocks = static_cast<int>(want < 16 * 148 ? want : 16 * 148);
  slot_count_kernel<false><<<blocks, kPackThreads, 0, s>>>(d, static_cast<int>(total));
  slot_scan_kernel<<<1, kScanThreads, 0, s>>>(d.first, static_cast<int>(bins));
  slot_count_kernel<true><<<blocks, kPackThreads, 0, s>>>(d, static_cast<int>(total));
  return cudaPeekAtLastError();
}

cudaError_t launch_gather_pack(cudaStream_t s, const GatherPackDev& g) {
  if (g.points <= 0) return cudaSuccess;
  if (g.slots_in > kMaxSlots) return cudaErrorInvalidValue;
  gather_pack_kernel<<<(g.points + kPackThreads - 1) / kPackThreads, kPackThreads, 0, s>>>(g);
  return cudaPeekAtLastError();
}

cudaError_t launch_voxel_histogram(cudaStream_t s, const uint8_t* v, int64_t n, int* counts) {
  cudaError_t err = cudaMemsetAsync(counts, 0, 256 * sizeof(int), s);
  if (err != cudaSuccess || n <= 0) return err;
  int blocks = static_cast<int>((n + kPackThreads - 1) / kPackThreads);
  if (blocks > 4 * 148) blocks = 4 * 148;
  voxel_histogram_kernel<<<blocks, kPackThreads, 0, s>>>(v, n, counts);
  return cudaPeekAtLastError();
}

}  // namespace fdtd
