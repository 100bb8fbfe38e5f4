// Device reductions behind automatic termination: field diagnostics
// (integrated energy, largest |field|, non-finite count) and the change of
// each DFT monitor vector between checks.
//
// beamz evaluates both between run chunks with jnp reductions
// (beamz/simulation/execute.py:184-222 _field_diagnostics, 294-316
// _relative_monitor_change, driven by run_until_terminated 1312-1484).  Here
// each is a bandwidth-bound read of the fields or the arena: coalesced row
// sweeps, float products with double accumulation across rows, warp-shuffle
// and shared-memory block reductions, and a fixed partition and summation
// order, so a result is identical from run to run.

#include <cooperative_groups.h>

#include "kernels.cuh"

namespace fdtd {

namespace {

constexpr int kDiagThreads = 256;
constexpr int kDiagWarps = kDiagThreads / 32;

__device__ __forceinline__ void warp_reduce(double& s, float& m, unsigned& n) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
    n += __shfl_down_sync(0xffffffffu, n, o);
  }
}

// Block reduction of (sum, max, count); the result is valid in thread 0.
__device__ __forceinline__ void block_reduce(double& s, float& m, unsigned& n) {
  __shared__ double ss[kDiagWarps];
  __shared__ float sm[kDiagWarps];
  __shared__ unsigned sn[kDiagWarps];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  warp_reduce(s, m, n);
  if (l == 0) {
    ss[w] = s;
    sm[w] = m;
    sn[w] = n;
  }
  __syncthreads();
  if (w == 0) {
    s = l < kDiagWarps ? ss[l] : 0.0;
    m = l < kDiagWarps ? sm[l] : 0.0f;
    n = l < kDiagWarps ? sn[l] : 0u;
    warp_reduce(s, m, n);
  }
}

// Rows (k, j) of one component, one warp per row: warp w of block b sweeps
// rows b * warps_per_block + w, then + all warps of the grid; its lanes stride
// along x.  A lane forms each product eps * v^2 in float and sums its products
// of a row in float; each row then enters the double accumulator once, weighted
// by its y/z factor, with the two end sites of an edge-aligned x axis taken at
// half weight.  MAT: 0 eps_r = 1, 1 codebook ids and table (in shared memory), 2
// per-site array.  Vec: rows start on 16 bytes (the pitched layout), so a lane
// takes four sites per load; the sweep is a plain read of the fields and ids,
// and with 4-byte loads and a table gather per site it took 443 us at 384 x 384 x
// 192 (1.0 GB with the ids read per component; 282 us now).
template <int MAT, bool Vec>
__device__ __forceinline__ void diag_rows(const DiagComp& q, const float* table, double& s, float& mx, unsigned& bad) {
  constexpr int N = Vec ? 4 : 1;
  const int rows = q.d.z * q.d.y;  // < 2^31: component arrays are validated below 2^31 elements
  const int lane = threadIdx.x & 31;
  const int step = gridDim.x * kDiagWarps;
  for (int r = blockIdx.x * kDiagWarps + (threadIdx.x >> 5); r < rows; r += step) {
    const int k = r / q.d.y, j = r - k * q.d.y;
    const int64_t base = k * q.plane + j * q.row;
    const float* f = q.field + base;
    float acc = 0.0f, ends = 0.0f;
#pragma unroll 4
    for (int i0 = lane * N; i0 < q.d.x; i0 += 32 * N) {
      float x[N];
      uint32_t id[N];
      if constexpr (Vec) {
        const float4 v = *reinterpret_cast<const float4*>(f + i0);
        x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
        if constexpr (MAT == 1) {
          const uint4 w = *reinterpret_cast<const uint4*>(q.ids + base + i0);
          id[0] = w.x, id[1] = w.y, id[2] = w.z, id[3] = w.w;
        }
      } else {
        x[0] = f[i0];
        if constexpr (MAT == 1) id[0] = q.ids[base + i0];
      }
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const int i = i0 + n;
        const bool in = !Vec || i < q.d.x;  // the row's padding holds anything
        float e = 1.0f;
        if constexpr (MAT == 1) e = table[(id[n] >> q.shift) & 0xffu];
        if constexpr (MAT == 2) e = in ? q.eps[static_cast<int64_t>(r) * q.d.x + i] : 0.0f;
        const bool ok = isfinite(x[n]);
        bad += in && !ok;
        const float v = in && ok ? x[n] : 0.0f;
        mx = fmaxf(mx, fabsf(v));
        const float prod = in && ok ? e * v * v : 0.0f;
        acc += prod;
        if (i == 0 || i == q.d.x - 1) ends += prod;
      }
    }
    double h = 1.0;
    if (q.integrate_z && q.edge_z && (k == 0 || k == q.d.z - 1)) h *= 0.5;
    if (q.edge_y && (j == 0 || j == q.d.y - 1)) h *= 0.5;
    s += h * (static_cast<double>(acc) - (q.edge_x ? 0.5 * static_cast<double>(ends) : 0.0));
  }
}

__global__ void __launch_bounds__(kDiagThreads) diag_partial_kernel(DiagArgs a) {
  __shared__ float table[256];
  const int c = blockIdx.y;
  double s = 0.0;
  float mx = 0.0f;
  unsigned bad = 0;
  if ((a.active >> c) & 1) {
    const DiagComp& q = a.comp[c];
    if (q.ids) {
      for (int e = threadIdx.x; e < 256; e += kDiagThreads) table[e] = q.table[e];
      __syncthreads();
    }
    const bool vec = q.row % 4 == 0 && q.plane % 4 == 0 && q.row >= (q.d.x + 3) / 4 * 4 &&
                     (reinterpret_cast<uintptr_t>(q.field) & 15) == 0 && (reinterpret_cast<uintptr_t>(q.ids) & 15) == 0;
    if (q.ids) vec ? diag_rows<1, true>(q, table, s, mx, bad) : diag_rows<1, false>(q, table, s, mx, bad);
    else if (q.eps) vec ? diag_rows<2, true>(q, table, s, mx, bad) : diag_rows<2, false>(q, table, s, mx, bad);
    else vec ? diag_rows<0, true>(q, table, s, mx, bad) : diag_rows<0, false>(q, table, s, mx, bad);
  }
  block_reduce(s, mx, bad);
  if (threadIdx.x == 0) {
    double* o = a.partials + (static_cast<int64_t>(c) * gridDim.x + blockIdx.x) * 3;
    o[0] = s;
    o[1] = mx;
    o[2] = bad;
  }
}

// One block per component: the partials in block order.
__global__ void __launch_bounds__(kDiagThreads) diag_final_kernel(const double* partials, int blocks, double* out) {
  const int c = blockIdx.x;
  double s = 0.0;
  float mx = 0.0f;
  unsigned bad = 0;
  for (int b = threadIdx.x; b < blocks; b += kDiagThreads) {
    const double* o = partials + (static_cast<int64_t>(c) * blocks + b) * 3;
    s += o[0];
    mx = fmaxf(mx, static_cast<float>(o[1]));
    bad += static_cast<unsigned>(o[2]);
  }
  block_reduce(s, mx, bad);
  if (threadIdx.x == 0) {
    out[c * 3 + 0] = s;
    out[c * 3 + 1] = mx;
    out[c * 3 + 2] = bad;
  }
}

// A cluster of eight blocks per (monitor, component, frequency): squared norms
// of the change, the current and the previous vector, then prev <- current.  The
// cluster's first block adds the blocks' sums in order.  (One block per vector
// left most SMs idle: 90 vectors of 60 k points took 134 us, now 32 us.)
constexpr int kChangeBlocks = 8;

__global__ void __cluster_dims__(kChangeBlocks, 1, 1) __launch_bounds__(kDiagThreads)
    dft_change_kernel(DftDev d, float* prev_re, float* prev_im, double* out) {
  __shared__ double total[3];
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int part = blockIdx.x % kChangeBlocks, key = blockIdx.x / kChangeBlocks;
  const int f = key % d.max_freqs, mc = key / d.max_freqs;
  const int m = mc / 6, c = mc % 6;
  const int* cnt = d.counts + 5 * m;
  const int nf = min(max(cnt[0], 0), d.max_freqs);
  const int np = min(max(cnt[1], 0), d.max_points);
  const int voff = cnt[3];
  double dd = 0.0, cc = 0.0, pp = 0.0;
  const bool on = d.masks[m * 6 + c] != 0.0f && f < nf && voff >= 0 &&
                  voff + static_cast<int64_t>(6) * nf * np <= d.arena_len;
  if (on) {
    const int64_t base = voff + (static_cast<int64_t>(c) * nf + f) * np;
    for (int p = part * kDiagThreads + threadIdx.x; p < np; p += kChangeBlocks * kDiagThreads) {
      const float re = d.re[base + p], im = d.im[base + p];
      const double dr = static_cast<double>(re) - prev_re[base + p], di = static_cast<double>(im) - prev_im[base + p];
      const double pr = prev_re[base + p], pi = prev_im[base + p];
      dd += dr * dr + di * di;
      cc += static_cast<double>(re) * re + static_cast<double>(im) * im;
      pp += pr * pr + pi * pi;
      prev_re[base + p] = re;
      prev_im[base + p] = im;
    }
  }
  // Three block sums in sequence; each total lands in thread 0's variable and
  // stays there through the later reductions.
  float unused = 0.0f;
  unsigned none = 0;
  block_reduce(dd, unused, none);
  __syncthreads();
  block_reduce(cc, unused, none);
  __syncthreads();
  block_reduce(pp, unused, none);
  if (threadIdx.x == 0) {
    total[0] = dd;
    total[1] = cc;
    total[2] = pp;
  }
  cluster.sync();
  if (part == 0 && threadIdx.x < 3) {
    double sum = 0.0;
    for (int b = 0; b < kChangeBlocks; ++b) sum += *cluster.map_shared_rank(&total[threadIdx.x], b);
    out[key * 3 + threadIdx.x] = sum;
  }
  cluster.sync();  // no block leaves while its sums are read
}

}  // namespace

cudaError_t launch_field_diagnostics(cudaStream_t s, const DiagArgs& a, double* out) {
  diag_partial_kernel<<<dim3(FDTD_DIAG_BLOCKS, 6, 1), kDiagThreads, 0, s>>>(a);
  cudaError_t err = cudaPeekAtLastError();
  if (err != cudaSuccess) return err;
  diag_final_kernel<<<6, kDiagThreads, 0, s>>>(a.partials, FDTD_DIAG_BLOCKS, out);
  return cudaPeekAtLastError();
}

cudaError_t launch_dft_change(cudaStream_t s, const DftDev& d, float* prev_re, float* prev_im, double* out) {
  const int keys = d.monitor_count * 6 * d.max_freqs;
  if (keys <= 0) return cudaSuccess;
  dft_change_kernel<<<keys * kChangeBlocks, kDiagThreads, 0, s>>>(d, prev_re, prev_im, out);
  return cudaPeekAtLastError();
}

}  // namespace fdtd
