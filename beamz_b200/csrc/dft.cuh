// The DFT accumulation of a batch of buffered steps, shared by the flush
// kernels (io.cu, block2d.cu).
#pragma once

#include "kernels.cuh"

namespace fdtd {

constexpr int kDftMaxFreqs = 64;
constexpr int kDftMaxBatch = 16;

struct FlushShared {
  float cosv[kDftMaxBatch][kDftMaxFreqs];
  float sinv[kDftMaxBatch][kDftMaxFreqs];
  float scale[kDftMaxBatch];
  float window[kDftMaxBatch];
  float time[kDftMaxBatch];
  int on[kDftMaxBatch];
};

// Adds `count` buffered steps (absolute steps counter + first ..) of one
// (monitor, component) to the arena in step order, for the points `p0` +
// thread; with `weights` also the monitor's window weight sums.  All threads of
// the block call it.  `samples` holds [batch, M, 6, P] interpolated values or,
// with Raw, [batch, M, 6, K, P] gathered field values, whose weighted sum is
// formed here in dft_gather's order (slots up to the first zero weight).  The
// gate, window, scale and phase of each step are dft_kernel's
// (beamz/simulation/observe.py:327-357, 529-585).
template <bool Raw>
__device__ void dft_flush_body(const DftDev& d, FlushShared& sh, const float* samples, const int* counter, int first,
                               int slot0, int count, int m, int c, int p0, bool weights, int tid, int nthreads) {
  const int* cnt = d.counts + 5 * m;
  const int nf = min(max(cnt[0], 0), d.max_freqs);
  const int np = min(max(cnt[1], 0), d.max_points);
  const int interval = cnt[2] > 0 ? cnt[2] : 1;
  const int voff = cnt[3], woff = cnt[4];
  const float t0 = d.windows[3 * m], t1 = d.windows[3 * m + 1], unit = d.windows[3 * m + 2];
  for (int s = tid; s < count; s += nthreads) {
    const int step = counter[0] + first + s;
    int ti = step < 0 ? 0 : step;
    ti = ti >= d.step_time_len ? d.step_time_len - 1 : ti;
    const float t = d.step_time[ti];
    const bool on = step % interval == 0 && t >= t0 && t <= t1;
    float window = 1.0f;
    if (on && d.codes[2 * m] == 1 && isfinite(t1) && t1 > t0) {
      const float span = fmaxf(t1 - t0, 1e-30f);
      const float tau = fminf(fmaxf((t - t0) / span, 0.0f), 1.0f);
      window = 0.5f * (1.0f - cosf(6.2831855f * tau));
    }
    float scale = fmaxf(window, 0.0f);
    if (d.codes[2 * m + 1] == 1) {
      const float phys = ((d.dt * static_cast<float>(interval)) * 299792458.0f) / unit;
      scale = scale * (phys / sqrtf(6.2831855f));
    }
    sh.on[s] = on ? 1 : 0;
    sh.scale[s] = scale;
    sh.window[s] = window;
    sh.time[s] = t;
  }
  __syncthreads();
  for (int e = tid; e < count * nf; e += nthreads) {
    const int s = e / nf, f = e % nf;
    const float theta = (6.2831855f * d.freqs[m * d.max_freqs + f]) * sh.time[s];
    float sn, cs;
    sincosf(theta, &sn, &cs);
    sh.cosv[s][f] = cs;
    sh.sinv[s][f] = sn;
  }
  __syncthreads();
  if (weights) {
    for (int f = tid; f < nf; f += nthreads) {
      if (woff < 0 || woff + f >= d.weight_len) continue;
      float ws = d.weight_sum[woff + f];
      for (int s = 0; s < count; ++s)
        if (sh.on[s]) ws += sh.window[s];
      d.weight_sum[woff + f] = ws;
    }
  }
  const float mask = d.masks[m * 6 + c];
  const int p = p0 + tid;
  if (p >= np || mask == 0.0f) return;
  if (voff < 0 || voff + static_cast<int64_t>(6) * nf * np > d.arena_len) return;
  const int64_t out = voff + (static_cast<int64_t>(c) * nf) * np + p;
  // The point's buffered samples are loaded once, and the arena words of
  // kFlushFreqs frequencies together, so a flush costs a few memory round
  // trips per point; each arena word still adds the steps in step order.
  constexpr int kFlushFreqs = 4;
  float vs[kDftMaxBatch];
  if constexpr (!Raw) {
    const int64_t stride = static_cast<int64_t>(d.monitor_count) * 6 * d.max_points;
    const float* v = samples + slot0 * stride + (static_cast<int64_t>(m) * 6 + c) * d.max_points + p;
#pragma unroll
    for (int s = 0; s < kDftMaxBatch; ++s) vs[s] = s < count && sh.on[s] ? v[s * stride] : 0.0f;
  } else {
    const int K = d.neighbors;
    const int64_t row = d.max_points, stride = static_cast<int64_t>(d.monitor_count) * 6 * K * row;
    const int64_t base = (static_cast<int64_t>(m) * 6 + c) * K * row + p;
    const float* v = samples + slot0 * stride + base;
#pragma unroll
    for (int s = 0; s < kDftMaxBatch; ++s) vs[s] = 0.0f;
    for (int n = 0; n < K; ++n) {
      const float w = d.weights[base + n * row];
      if (w == 0.0f) break;
      const int idx = d.indices[base + n * row];
      if (idx < 0 || idx >= d.field_len[c]) continue;
#pragma unroll
      for (int s = 0; s < kDftMaxBatch; ++s)
        if (s < count && sh.on[s]) vs[s] = vs[s] + v[s * stride + n * row] * w;
    }
  }
  for (int f0 = 0; f0 < nf; f0 += kFlushFreqs) {
    float re[kFlushFreqs], im[kFlushFreqs];
#pragma unroll
    for (int q = 0; q < kFlushFreqs; ++q) {
      const int64_t o = out + static_cast<int64_t>(f0 + q) * np;
      re[q] = f0 + q < nf ? d.re[o] : 0.0f;
      im[q] = f0 + q < nf ? d.im[o] : 0.0f;
    }
#pragma unroll
    for (int q = 0; q < kFlushFreqs; ++q) {
      const int f = f0 + q;
      if (f >= nf) break;
#pragma unroll
      for (int s = 0; s < kDftMaxBatch; ++s) {
        if (s >= count) break;
        if (!sh.on[s]) continue;
        const float sm = sh.scale[s] * mask;
        re[q] += sm * (sh.cosv[s][f] * vs[s]);
        im[q] += sm * (sh.sinv[s][f] * vs[s]);
      }
      const int64_t o = out + static_cast<int64_t>(f) * np;
      d.re[o] = re[q];
      d.im[o] = im[q];
    }
  }
}

}  // namespace fdtd
