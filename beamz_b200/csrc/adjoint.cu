// Discrete adjoint of the leapfrog step (dense layout, per-site E material).
//
// The step without its sources is linear in the state u = (E, H, psi_H,
// psi_E); the adjoint applies the exact transpose of each of its linear maps
// in reverse order (beamz/simulation/execute.py:467-541 gives the forward
// order):
//
//   forward step n                      adjoint step n (on lambda)
//   1. H <- mask_H (dec H - src curl'E)  5. DFT source: lambda += dJ/du_{n+1}
//   2. E <- mask_E (E + c curl'H)        4. E transpose (per E site, then
//   3. DFT of u_{n+1}                       Bx^T gather per H site)
//                                        3. H transpose (per H site, then
//                                           D^T gather per E site)
//
// where curl' sums the CPML-corrected derivatives d' of each term
// (psi' = b psi + a d, d' = d / kappa + psi'; beamz/simulation/kernels.py:
// 257-264), D is the forward difference E -> H and B the ghost-padded
// backward difference H -> E (zero ghost on a metallic face, edge copy
// elsewhere; beamz/lattice.py:523-551).  Transposes:
//   CPML:  acc = lam_psi' + lam_d';  lam_psi = b acc;  lam_d = lam_d' / kappa + a acc
//   D^T:   (D^T u)[m] = (u[m-1] - u[m]) / res   (u outside [0, N) is zero)
//   B^T:   (B^T t)[h] = (r(h) t[h] - r(h+1) t[h+1]) / res, r(m) = 1 for the
//          rows of B that difference two samples or a metallic ghost, 0 for
//          the rows whose edge-copy ghost makes them zero.
//   With derivative metrics (axis-uniform / rectilinear grids) each
//   difference carries its coordinate's inverse distance instead of 1/res:
//   (D^T u)[m] = mh[m-1] u[m-1] - mh[m] u[m] and
//   (B^T t)[h] = r(h) me[h] t[h] - r(h+1) me[h+1] t[h+1].
// Every lambda_d is recomputed where it is gathered, from the adjoint fields,
// the coefficients and the memories of its site (a handful of L1 / L2 hits),
// instead of travelling through one scratch array per term: a step is three
// kernels.  The H pass reads the E adjoint fields, the E pass the new H ones,
// each writing only its own sites, and each set of memories is updated when its
// last reader is done (psi_E by the E pass, psi_H by the third kernel, over the
// absorber slabs alone).  With scratch and one launch per component and pass, a
// 256 x 256 x 128 step moved 1.7 GB in twelve launches; these two passes 0.86 GB.  The
// permittivity gradient accumulates mu * curl'_n per E site over a design box,
// mu = the masked E adjoint and curl'_n the forward curl.

#include "kernels.cuh"

namespace fdtd {

namespace {

// Term tables (3D order: H 0 Hx-y, 1 Hx-z, 2 Hy-z, 3 Hy-x, 4 Hz-x, 5 Hz-y;
// E likewise for Ex, Ey, Ez; even terms enter with +, odd with -).
// The kernels take their component as a template argument, so that these
// lookups (and the term loops of the gathers) resolve at compile time.
__host__ __device__ constexpr int adj_h_src(int t) { return 2 - t % 3; }  // E component an H term differentiates
__host__ __device__ constexpr int adj_e_src(int t) { return 5 - t % 3; }  // H component an E term differentiates
// Axis of term t's derivative, for H and E terms alike: 1, 0, 0, 2, 2, 1.
__host__ __device__ constexpr int adj_axis(int t) { return (t == 0 || t == 5) ? 1 : ((t == 1 || t == 2) ? 0 : 2); }

constexpr int kAdjThreads = 256;

// Element offsets fit 32 bits (every entry point validates arrays below 2^31
// elements).
__device__ __forceinline__ int at(const Dims& d, int k, int j, int i) { return (k * d.y + j) * d.x + i; }

__device__ __forceinline__ int coord_of(int axis, int k, int j, int i) { return axis == 0 ? k : (axis == 1 ? j : i); }

__device__ __forceinline__ int psi_index(const CpmlTermDev& t, int axis, int slot, int k, int j, int i) {
  const int pk = axis == 0 ? slot : k, pj = axis == 1 ? slot : j, pi = axis == 2 ? slot : i;
  return (pk * t.pdy + pj) * t.pdx + pi;
}

__device__ __forceinline__ float coef_at(const float* p, int full, int idx) { return p[full ? idx : 0]; }

// Transpose of one CPML-corrected derivative at a site: lam_d' -> lam_d from the
// adjoint memory (held in psi_out), which stays as it is (Update: advances).
template <bool Update>
__device__ __forceinline__ float cpml_transpose(const CpmlTermDev& t, int axis, int k, int j, int i, float ld) {
  const int slot = cpml_slot(t, coord_of(axis, k, j, i));
  if (slot < 0) return ld;
  const int off = psi_index(t, axis, slot, k, j, i);
  const float acc = t.psi_out[off] + ld;
  if (Update) t.psi_out[off] = t.b[slot] * acc;
  return t.k[slot] * ld + t.a[slot] * acc;
}

// Per axis: is this lattice point, with its neighbours one cell up and down, off
// both faces and outside every slab?  Then the axis's terms need no ghost or
// memory test.
struct InnerAxes {
  bool in[3];
};
__device__ __forceinline__ InnerAxes inner_axes(const Step3D& p, int k, int j, int i) {
  auto in = [&](int axis, int c, int n) {
    return c >= 1 && c <= n - 2 && c - 1 >= p.cpml_inner[axis][0] && c + 1 < p.cpml_inner[axis][1];
  };
  return {{in(0, k, p.Z), in(1, j, p.Y), in(2, i, p.X)}};
}

// The lattice points of a launch: a block covers 64 x 4 points of one plane, so
// that z and y (and with them most slab tests) are uniform over a warp.  Written
// term by term, with every site's offset, ghost, mask and slot test between its
// loads, the passes issued 750-880 instructions per warp of points at 0.7 per
// cycle (252 + 302 us at 256 x 256 x 128).  Here each site is read once, all
// loads go out before the first test, and only the terms of an axis whose slab or
// face is near are looked at further: 197 + 288 us.  What is left is the latency
// of the slab points' chains, so the registers are held to eight blocks per SM
// (at five: 192 + 345 us, at three: E pass 511 us).
constexpr int kAdjX = 64, kAdjY = 4;

// 4b + mask of 3a, per H site: lambda_H += B^T lam_d, then the PEC mask.
template <int Active, bool Metric>
__device__ __forceinline__ void h_point(const Step3D& p, const AdjDev& a, float inv_res, int k, int j, int i) {
  constexpr bool EX = Active & 1, EY = Active & 2, EZ = Active & 4, HX = Active & 8, HY = Active & 16, HZ = Active & 32;
  const int Z = p.Z, Y = p.Y, X = p.X;
  const bool kz = k < Z, jy = j < Y, ix = i < X;  // is there a neighbour one cell up?
  const int nx = X + 1, ny = Y + 1;
  const int ox = (k * ny + j) * X + i, oy = (k * Y + j) * nx + i, oz = (k * ny + j) * nx + i;
  const int px = ny * X, py = Y * nx;  // planes of Ex (and Hy), Ey (and Hx)
  // Every load first (at offset 0 where a site does not exist), with nothing that
  // could branch between them; then masks and products.
  struct Site {
    float lam, src;
  };
  auto load = [&](int c, bool ok, int o) -> Site {
    const int at = ok ? o : 0;
    return {a.lam[c][at], coef_at(p.em.source[c], p.em.source_full[c], at)};
  };
  Site sx0{}, sxz{}, sxy{}, sy0{}, syz{}, syx{}, sz0{}, szy{}, szx{};
  if constexpr (EX) {
    sx0 = load(0, ix, ox);
    if constexpr (HY) sxz = load(0, ix && kz, ox + px);
    if constexpr (HZ) sxy = load(0, ix && jy, ox + X);
  }
  if constexpr (EY) {
    sy0 = load(1, jy, oy);
    if constexpr (HX) syz = load(1, jy && kz, oy + py);
    if constexpr (HZ) syx = load(1, jy && ix, oy + 1);
  }
  if constexpr (EZ) {
    sz0 = load(2, kz, oz);
    if constexpr (HX) szy = load(2, kz && jy, oz + nx);
    if constexpr (HY) szx = load(2, kz && ix, oz + 1);
  }
  const int oh = (k * Y + j) * X + i;                                 // Hz (Z + 1, Y, X)
  const float lx = HX ? a.lam[3][kz && jy ? oy : 0] : 0.0f;           // Hx (Z, Y, X + 1): Ey's rows and planes
  const float ly = HY ? a.lam[4][kz && ix ? ox : 0] : 0.0f;           // Hy (Z, Y + 1, X): Ex's
  const float lz = HZ ? a.lam[5][jy && ix ? oh : 0] : 0.0f;
  if (p.metallic) {
    auto mask = [&](int c, Site& v, int kk, int jj, int ii) {
      if (e_constrained(p.metallic, c, component_dims(c, Z, Y, X), kk, jj, ii)) v.lam = 0.0f;
    };
    mask(0, sx0, k, j, i), mask(0, sxz, k + 1, j, i), mask(0, sxy, k, j + 1, i);
    mask(1, sy0, k, j, i), mask(1, syz, k + 1, j, i), mask(1, syx, k, j, i + 1);
    mask(2, sz0, k, j, i), mask(2, szy, k, j + 1, i), mask(2, szx, k, j, i + 1);
  }
  // source * mask * lambda_E.
  const float x0 = sx0.src * sx0.lam, xz = sxz.src * sxz.lam, xy = sxy.src * sxy.lam;
  const float y0 = sy0.src * sy0.lam, yz = syz.src * syz.lam, yx = syx.src * syx.lam;
  const float z0 = sz0.src * sz0.lam, zy = szy.src * szy.lam, zx = szx.src * szx.lam;
  const InnerAxes in = inner_axes(p, k, j, i);
  // lam_d of E term t at a site from its product, and 0 where the ghost makes B's
  // row vanish.
  auto ld = [&](int t, float v, int kk, int jj, int ii) -> float {
    const int axis = adj_axis(t);
    if (in.in[axis]) return v;
    const int r = coord_of(axis, kk, jj, ii), N = axis == 0 ? Z : (axis == 1 ? Y : X);
    if (!((r >= 1 && r <= N - 1) || (r == 0 && wall(p.metallic, axis, false)) || (r == N && wall(p.metallic, axis, true))))
      return 0.0f;
    return p.cpml ? cpml_transpose<false>(p.et[t], axis, kk, jj, ii, v) : v;
  };
  // Derivative metrics: the backward difference at E coordinate m was scaled by
  // metric_e[m] (and the ghost rows by metric_e[0] / [N]).
  auto gather = [&](int t, float t0, float t1) -> float {
    if constexpr (Metric) {
      const int axis = adj_axis(t), m = coord_of(axis, k, j, i);
      return t0 * p.metric_e[axis][m] - t1 * p.metric_e[axis][m + 1];
    } else {
      return (t0 - t1) * inv_res;
    }
  };
  if constexpr (HX) {
    if (kz && jy) {
      float acc = 0.0f;
      if constexpr (EY) acc += gather(2, ld(2, y0, k, j, i), ld(2, yz, k + 1, j, i));
      if constexpr (EZ) acc += gather(5, ld(5, -z0, k, j, i), ld(5, -zy, k, j + 1, i));
      float v = lx + acc;
      if (p.metallic && h_constrained(p.metallic, 3, component_dims(3, Z, Y, X), k, j, i)) v = 0.0f;
      a.lam[3][oy] = v;
    }
  }
  if constexpr (HY) {
    if (kz && ix) {
      float acc = 0.0f;
      if constexpr (EX) acc += gather(1, ld(1, -x0, k, j, i), ld(1, -xz, k + 1, j, i));
      if constexpr (EZ) acc += gather(4, ld(4, z0, k, j, i), ld(4, zx, k, j, i + 1));
      float v = ly + acc;
      if (p.metallic && h_constrained(p.metallic, 4, component_dims(4, Z, Y, X), k, j, i)) v = 0.0f;
      a.lam[4][ox] = v;
    }
  }
  if constexpr (HZ) {
    if (jy && ix) {
      float acc = 0.0f;
      if constexpr (EX) acc += gather(0, ld(0, x0, k, j, i), ld(0, xy, k, j + 1, i));
      if constexpr (EY) acc += gather(3, ld(3, -y0, k, j, i), ld(3, -yx, k, j, i + 1));
      float v = lz + acc;
      if (p.metallic && h_constrained(p.metallic, 5, component_dims(5, Z, Y, X), k, j, i)) v = 0.0f;
      a.lam[5][oh] = v;
    }
  }
}

// 4a + 3b, per E site: mask, memories and identity part of the E transpose, the
// design-box gradient, then lambda_E += D^T lam_d.
template <int Active, bool Metric>
__device__ __forceinline__ void e_point(const Step3D& p, const AdjDev& a, float inv_res, int k, int j, int i) {
  constexpr bool EX = Active & 1, EY = Active & 2, EZ = Active & 4, HX = Active & 8, HY = Active & 16, HZ = Active & 32;
  const int Z = p.Z, Y = p.Y, X = p.X;
  const bool kz = k < Z, jy = j < Y, ix = i < X;     // is the point inside the H extent of an axis?
  const bool kd = k >= 1, jd = j >= 1, id = i >= 1;  // is there a neighbour one cell down?
  const int nx = X + 1, ny = Y + 1;
  const int ox = (k * ny + j) * X + i, oy = (k * Y + j) * nx + i, oz = (k * ny + j) * nx + i, oh = (k * Y + j) * X + i;
  const int px = ny * X, py = Y * nx;
  // Every load first, as in h_point: source * lambda_H of the sites (masked by the
  // H pass; 0 where there is none) and the own E values.
  auto prod = [&](int h, bool ok, int o) -> float {
    const int at = ok ? o : 0;
    const float v = coef_at(p.hm.source[h], p.hm.source_full[h], at) * a.lam[3 + h][at];
    return ok ? v : 0.0f;
  };
  const float ex = EX ? a.lam[0][ix ? ox : 0] : 0.0f, ey = EY ? a.lam[1][jy ? oy : 0] : 0.0f;
  const float ez = EZ ? a.lam[2][kz ? oz : 0] : 0.0f;
  const float dx = EX ? coef_at(p.em.decay[0], p.em.decay_full[0], ix ? ox : 0) : 0.0f;
  const float dy = EY ? coef_at(p.em.decay[1], p.em.decay_full[1], jy ? oy : 0) : 0.0f;
  const float dz = EZ ? coef_at(p.em.decay[2], p.em.decay_full[2], kz ? oz : 0) : 0.0f;
  float x0 = 0.f, xz = 0.f, xy = 0.f, y0 = 0.f, yz = 0.f, yx = 0.f, z0 = 0.f, zy = 0.f, zx = 0.f;
  if constexpr (HX) {
    x0 = prod(0, kz && jy, oy);
    if constexpr (EY) xz = prod(0, kd && jy, oy - py);
    if constexpr (EZ) xy = prod(0, kz && jd, oy - nx);
  }
  if constexpr (HY) {
    y0 = prod(1, kz && ix, ox);
    if constexpr (EX) yz = prod(1, kd && ix, ox - px);
    if constexpr (EZ) yx = prod(1, kz && id, ox - 1);
  }
  if constexpr (HZ) {
    z0 = prod(2, jy && ix, oh);
    if constexpr (EX) zy = prod(2, jd && ix, oh - X);
    if constexpr (EY) zx = prod(2, jy && id, oh - 1);
  }
  const InnerAxes in = inner_axes(p, k, j, i);
  const bool in_box = k >= a.box_lo[0] && k < a.box_hi[0] && j >= a.box_lo[1] && j < a.box_hi[1] && i >= a.box_lo[2] &&
                      i < a.box_hi[2];
  // lam_d of H term t at a site from its product (0 outside the H extent).
  auto ld = [&](int t, float v, bool ok, int kk, int jj, int ii) -> float {
    const int axis = adj_axis(t);
    if (in.in[axis] || !p.cpml || !ok) return v;
    return cpml_transpose<false>(p.ht[t], axis, kk, jj, ii, v);
  };
  // Derivative metrics: the forward difference at H coordinate m was scaled by
  // metric_h[m].
  auto gather = [&](int t, float prev, bool has_prev, float here, bool has_here) -> float {
    if constexpr (Metric) {
      const int axis = adj_axis(t), m = coord_of(axis, k, j, i);
      return (has_prev ? prev * p.metric_h[axis][m - 1] : 0.0f) - (has_here ? here * p.metric_h[axis][m] : 0.0f);
    } else {
      return (prev - here) * inv_res;
    }
  };
  // One E component: identity part, gather, memories, gradient.
  auto site = [&](int c, int o, float mu, float dec, float acc) {
    if (p.metallic && e_constrained(p.metallic, c, component_dims(c, Z, Y, X), k, j, i)) mu = 0.0f;
    a.lam[c][o] = dec * mu + acc;
    if (p.cpml) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int t = 2 * c + s, axis = adj_axis(t);
        if (in.in[axis] || !((Active >> adj_e_src(t)) & 1) || cpml_slot(p.et[t], coord_of(axis, k, j, i)) < 0) continue;
        const float src = coef_at(p.em.source[c], p.em.source_full[c], o);
        cpml_transpose<true>(p.et[t], axis, k, j, i, (s == 0 ? src : -src) * mu);
      }
    }
    if (in_box && a.grad[c] != nullptr) {
      const int64_t b = (static_cast<int64_t>(k - a.box_lo[0]) * (a.box_hi[1] - a.box_lo[1]) + (j - a.box_lo[1])) *
                            (a.box_hi[2] - a.box_lo[2]) +
                        (i - a.box_lo[2]);
      a.grad[c][b] += mu * a.curl[c][b];
    }
  };
  if constexpr (EX) {
    if (ix) {
      float acc = 0.0f;
      if constexpr (HY) acc += gather(2, ld(2, -yz, kd, k - 1, j, i), kd, ld(2, -y0, kz, k, j, i), kz);
      if constexpr (HZ) acc += gather(5, ld(5, zy, jd, k, j - 1, i), jd, ld(5, z0, jy, k, j, i), jy);
      site(0, ox, ex, dx, acc);
    }
  }
  if constexpr (EY) {
    if (jy) {
      float acc = 0.0f;
      if constexpr (HX) acc += gather(1, ld(1, xz, kd, k - 1, j, i), kd, ld(1, x0, kz, k, j, i), kz);
      if constexpr (HZ) acc += gather(4, ld(4, -zx, id, k, j, i - 1), id, ld(4, -z0, ix, k, j, i), ix);
      site(1, oy, ey, dy, acc);
    }
  }
  if constexpr (EZ) {
    if (kz) {
      float acc = 0.0f;
      if constexpr (HX) acc += gather(0, ld(0, -xy, jd, k, j - 1, i), jd, ld(0, -x0, jy, k, j, i), jy);
      if constexpr (HY) acc += gather(3, ld(3, yx, id, k, j, i - 1), id, ld(3, y0, ix, k, j, i), ix);
      site(2, oz, ez, dz, acc);
    }
  }
}

// Blocks stride over rows and planes beyond the launch limits; a 2D program lives
// on plane 0.
template <int Active, bool Metric>
__global__ void __launch_bounds__(kAdjX* kAdjY, 8) adj_h_pass(const __grid_constant__ Step3D p,
                                                              const __grid_constant__ AdjDev a) {
  const int i = blockIdx.x * kAdjX + threadIdx.x;
  if (i > p.X) return;
  const float inv_res = 1.0f / p.res;
  const int planes = Active == kActive3D ? p.Z + 1 : 1;
#pragma unroll 1
  for (int k = blockIdx.z; k < planes; k += gridDim.z)
#pragma unroll 1
    for (int j = blockIdx.y * kAdjY + threadIdx.y; j <= p.Y; j += gridDim.y * kAdjY)
      h_point<Active, Metric>(p, a, inv_res, k, j, i);
}

template <int Active, bool Metric>
__global__ void __launch_bounds__(kAdjX* kAdjY, 8) adj_e_pass(const __grid_constant__ Step3D p,
                                                              const __grid_constant__ AdjDev a) {
  const int i = blockIdx.x * kAdjX + threadIdx.x;
  if (i > p.X) return;
  const float inv_res = 1.0f / p.res;
  const int planes = Active == kActive3D ? p.Z + 1 : 1;
#pragma unroll 1
  for (int k = blockIdx.z; k < planes; k += gridDim.z)
#pragma unroll 1
    for (int j = blockIdx.y * kAdjY + threadIdx.y; j <= p.Y; j += gridDim.y * kAdjY)
      e_point<Active, Metric>(p, a, inv_res, k, j, i);
}

// The rest of 3a, per H component (blockIdx.y): the memories, over the slabs;
// and, where the H decay is not exactly 1, over every site with its scaling.
template <int Active>
__global__ void __launch_bounds__(kAdjThreads) adj_h_finish(const __grid_constant__ Step3D p,
                                                            const __grid_constant__ AdjDev a) {
  // Unsigned: a component may hold 2^31 - 1 elements, and the last stride passes that.
  const unsigned first = blockIdx.x * kAdjThreads + threadIdx.x, stride = gridDim.x * kAdjThreads;
#pragma unroll
  for (int hc = 0; hc < 3; ++hc) {
    if (!((Active >> (3 + hc)) & 1) || static_cast<int>(blockIdx.y) != hc) continue;
    const Dims d = component_dims(3 + hc, p.Z, p.Y, p.X);
    auto advance = [&](int t, int k, int j, int i, float mu) {
      const float src = coef_at(p.hm.source[hc], p.hm.source_full[hc], at(d, k, j, i));
      cpml_transpose<true>(p.ht[t], adj_axis(t), k, j, i, (t % 2 == 0 ? -src : src) * mu);
    };
    const bool scaled = p.hm.decay_full[hc] || p.hm.decay[hc][0] != 1.0f;
    if (!scaled) {
      if (!p.cpml) continue;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int t = 2 * hc + s, axis = adj_axis(t);
        if (!((Active >> adj_h_src(t)) & 1)) continue;
        const CpmlTermDev& term = p.ht[t];
        const int w = term.low + term.high;
        if (w == 0) continue;
        const Dims sd = {axis == 0 ? w : d.z, axis == 1 ? w : d.y, axis == 2 ? w : d.x};  // the slab
        const unsigned n = sd.z * sd.y * sd.x;
        for (unsigned e = first; e < n; e += stride) {
          const int r = e / sd.x;
          int i = e - r * sd.x, k = r / sd.y, j = r - k * sd.y;
          int& x = axis == 0 ? k : (axis == 1 ? j : i);
          if (x >= term.low) x += term.n_axis - w;  // high slots
          advance(t, k, j, i, a.lam[3 + hc][at(d, k, j, i)]);
        }
      }
      continue;
    }
    const unsigned n = d.z * d.y * d.x;
    for (unsigned e = first; e < n; e += stride) {
      const int r = e / d.x;
      const int i = e - r * d.x, k = r / d.y, j = r - k * d.y;
      const float mu = a.lam[3 + hc][e];
      if (p.cpml) {
#pragma unroll
        for (int s = 0; s < 2; ++s)
          if ((Active >> adj_h_src(2 * hc + s)) & 1) advance(2 * hc + s, k, j, i, mu);
      }
      a.lam[3 + hc][e] = coef_at(p.hm.decay[hc], p.hm.decay_full[hc], e) * mu;
    }
  }
}

// 5. DFT adjoint source for the sample at absolute step `step`:
// lambda[c][idx_k] += w_k * sum_f s (g_re cos(theta_f) + g_im sin(theta_f)),
// the transpose of the accumulation in io.cu (observe.py:529-585).
constexpr int kAdjMaxFreqs = 64;

__global__ void __launch_bounds__(kAdjThreads) adj_dft_kernel(DftDev d, AdjDev a, int step) {
  const int mc = blockIdx.y;
  const int m = mc / 6, c = mc % 6;
  const int* cnt = d.counts + 5 * m;
  const int nf = min(max(cnt[0], 0), d.max_freqs);
  const int np = min(max(cnt[1], 0), d.max_points);
  const int interval = cnt[2] > 0 ? cnt[2] : 1;
  const int voff = cnt[3];
  if (step % interval != 0 || a.lam[c] == nullptr) return;
  int ti = step < 0 ? 0 : step;
  ti = ti >= d.step_time_len ? d.step_time_len - 1 : ti;
  const float t = d.step_time[ti];
  const float t0 = d.windows[3 * m], t1 = d.windows[3 * m + 1], unit = d.windows[3 * m + 2];
  if (!(t >= t0 && t <= t1)) return;
  __shared__ float s_cos[kAdjMaxFreqs], s_sin[kAdjMaxFreqs];
  __shared__ float s_scale;
  if (threadIdx.x == 0) {
    float window = 1.0f;
    if (d.codes[2 * m] == 1 && isfinite(t1) && t1 > t0) {
      const float span = fmaxf(t1 - t0, 1e-30f);
      const float tau = fminf(fmaxf((t - t0) / span, 0.0f), 1.0f);
      window = 0.5f * (1.0f - cosf(6.2831855f * tau));
    }
    float scale = fmaxf(window, 0.0f);
    if (d.codes[2 * m + 1] == 1) {
      const float phys = ((d.dt * static_cast<float>(interval)) * 299792458.0f) / unit;
      scale = scale * (phys / sqrtf(6.2831855f));
    }
    s_scale = scale;
  }
  for (int f = threadIdx.x; f < nf; f += blockDim.x) {
    const float theta = (6.2831855f * d.freqs[m * d.max_freqs + f]) * t;
    float sn, cs;
    sincosf(theta, &sn, &cs);
    s_cos[f] = cs;
    s_sin[f] = sn;
  }
  __syncthreads();
  const float mask = d.masks[m * 6 + c];
  const int pidx = blockIdx.x * blockDim.x + threadIdx.x;
  if (pidx >= np || mask == 0.0f) return;
  if (voff < 0 || voff + static_cast<int64_t>(6) * nf * np > d.arena_len) return;
  const int64_t out = voff + (static_cast<int64_t>(c) * nf) * np + pidx;
  float g = 0.0f;
  for (int f = 0; f < nf; ++f) {
    const int64_t o = out + static_cast<int64_t>(f) * np;
    g += a.dft_grad_re[o] * s_cos[f] + a.dft_grad_im[o] * s_sin[f];
  }
  g *= s_scale * mask;
  if (g == 0.0f) return;
  const int64_t base = ((static_cast<int64_t>(m) * 6 + c) * d.neighbors) * d.max_points + pidx;
  for (int nb = 0; nb < d.neighbors; ++nb) {
    const float w = d.weights[base + static_cast<int64_t>(nb) * d.max_points];
    if (w == 0.0f) break;
    const int idx = d.indices[base + static_cast<int64_t>(nb) * d.max_points];
    if (idx >= 0 && idx < d.field_len[c]) atomicAdd(a.lam[c] + idx, w * g);
  }
}

// Forward curl of E component c over the design box from the current H
// (interior sites: plain differences, no ghost and no CPML; validated).
__global__ void __launch_bounds__(kAdjThreads) adj_curl_kernel(Step3D p, AdjDev a, int c) {
  const int bz = a.box_hi[0] - a.box_lo[0], by = a.box_hi[1] - a.box_lo[1], bx = a.box_hi[2] - a.box_lo[2];
  const int64_t n = static_cast<int64_t>(bz) * by * bx;
  const float res = p.res;
  const Dims lattice = {p.Z + 1, p.Y + 1, p.pitch};  // per-site programs on the pitched layout
  const Dims dx = p.site ? lattice : component_dims(3, p.Z, p.Y, p.X);
  const Dims dy = p.site ? lattice : component_dims(4, p.Z, p.Y, p.X);
  const Dims dz = p.site ? lattice : component_dims(5, p.Z, p.Y, p.X);
  for (int64_t b = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; b < n;
       b += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int i = a.box_lo[2] + static_cast<int>(b % bx);
    const int j = a.box_lo[1] + static_cast<int>((b / bx) % by);
    const int k = a.box_lo[0] + static_cast<int>(b / (static_cast<int64_t>(bx) * by));
    const float* Hx = p.hin[0];
    const float* Hy = p.hin[1];
    const float* Hz = p.hin[2];
    // A backward difference along `axis` at E coordinate `at`: divided by the
    // cell size, or times the derivative metric there.
    auto sc = [&](float diff, int axis, int at) {
      const float* me = p.metric_e[axis];
      return me != nullptr ? diff * me[at] : diff / res;
    };
    float curl;
    if (c == 0) {
      curl = sc(Hz[lin(dz, k, j, i)] - Hz[lin(dz, k, j - 1, i)], 1, j);
      if (Hy) curl -= sc(Hy[lin(dy, k, j, i)] - Hy[lin(dy, k - 1, j, i)], 0, k);
    } else if (c == 1) {
      curl = -sc(Hz[lin(dz, k, j, i)] - Hz[lin(dz, k, j, i - 1)], 2, i);
      if (Hx) curl += sc(Hx[lin(dx, k, j, i)] - Hx[lin(dx, k - 1, j, i)], 0, k);
    } else {
      curl = sc(Hy[lin(dy, k, j, i)] - Hy[lin(dy, k, j, i - 1)], 2, i) -
             sc(Hx[lin(dx, k, j, i)] - Hx[lin(dx, k, j - 1, i)], 1, j);
    }
    a.curl[c][b] = curl;
  }
}

// Grid-stride launches of 16 blocks per SM: each thread then takes a few
// dozen elements of a large component rather than one, so block scheduling
// does not dominate these short per-element passes.
unsigned blocks_for(int64_t n) {
  int dev = 0, sms = 0;  // the current device's SM count (a cheap attribute query)
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      sms <= 0)
    sms = 148;
  const int64_t b = (n + kAdjThreads - 1) / kAdjThreads;
  const int64_t cap = static_cast<int64_t>(sms) * 16;
  return static_cast<unsigned>(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

namespace {

template <int Active>
void launch_passes(cudaStream_t s, const Step3D& p, const AdjDev& a) {
  const auto capped = [](int n) { return static_cast<unsigned>(n < 65535 ? n : 65535); };
  const dim3 grid((p.X + kAdjX) / kAdjX, capped((p.Y + kAdjY) / kAdjY), Active != kActive3D ? 1 : capped(p.Z + 1));
  const dim3 block(kAdjX, kAdjY, 1);
  if (has_metric(p)) {
    adj_h_pass<Active, true><<<grid, block, 0, s>>>(p, a);
    adj_e_pass<Active, true><<<grid, block, 0, s>>>(p, a);
  } else {
    adj_h_pass<Active, false><<<grid, block, 0, s>>>(p, a);
    adj_e_pass<Active, false><<<grid, block, 0, s>>>(p, a);
  }
  // The slabs hold a few per cent of the sites.
  const int64_t sites = static_cast<int64_t>(p.Z + 1) * (p.Y + 1) * (p.X + 1);
  adj_h_finish<Active><<<dim3(blocks_for(sites / 4), 3, 1), kAdjThreads, 0, s>>>(p, a);
}

}  // namespace

cudaError_t launch_adjoint_steps(cudaStream_t s, const Step3D& p, const DftDev* dft, AdjDev a, int active, int step,
                                 int count, int64_t curl_stride) {
  const bool source = dft != nullptr && dft->monitor_count > 0 && dft->max_points > 0 && a.dft_grad_re != nullptr;
  if (source && dft->max_freqs > kAdjMaxFreqs) return cudaErrorInvalidValue;
  for (int n = 0; n < count; ++n) {
    if (source) {
      const dim3 grid((dft->max_points + kAdjThreads - 1) / kAdjThreads, dft->monitor_count * 6, 1);
      adj_dft_kernel<<<grid, kAdjThreads, 0, s>>>(*dft, a, step - n);
    }
    switch (active) {
      case kActive3D: launch_passes<kActive3D>(s, p, a); break;
      case kActiveTM: launch_passes<kActiveTM>(s, p, a); break;
      default: launch_passes<kActiveTE>(s, p, a); break;
    }
    const cudaError_t err = cudaPeekAtLastError();
    if (err != cudaSuccess) return err;
    for (int c = 0; c < 3; ++c)
      if (a.curl[c] != nullptr) a.curl[c] -= curl_stride;
  }
  return cudaSuccess;
}

cudaError_t launch_adjoint_curl(cudaStream_t s, const Step3D& p, const AdjDev& a, int active) {
  const int64_t n = static_cast<int64_t>(a.box_hi[0] - a.box_lo[0]) * (a.box_hi[1] - a.box_lo[1]) *
                    (a.box_hi[2] - a.box_lo[2]);
  if (n <= 0) return cudaSuccess;
  for (int c = 0; c < 3; ++c) {
    if (!((active >> c) & 1) || a.curl[c] == nullptr) continue;
    adj_curl_kernel<<<blocks_for(n), kAdjThreads, 0, s>>>(p, a, c);
  }
  return cudaPeekAtLastError();
}

}  // namespace fdtd
