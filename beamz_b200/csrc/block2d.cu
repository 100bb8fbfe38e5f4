// Several 2D leapfrog steps in one launch (temporal blocking).
//
// A 2D grid is small: its fields live in L2, and one launch per step is bound
// by launch gaps and by the latency of loading a tile, two barriers and storing
// it again, not by arithmetic or bandwidth (400 x 400 cells: 10.5 us of device
// time and two launches per step for 1.9 MB of fields).  Here a CTA loads its
// tile with a halo of T cells, advances T steps in shared memory -- the
// correct region shrinks by one cell per side and step, and ends as the tile
// -- and stores once.  A CTA covers 64 columns (64 - 2T of them its own) by as
// many rows as put one CTA on every SM (TY own rows; two per SM on grids whose
// tiles would not leave room for a second one).  The steps are bound by
// instruction issue, so a thread owns four neighbouring columns: shared memory
// moves in 16-byte vectors, x neighbours come by shuffle, and the index and
// boundary work is paid once per four cells.  Halo cells are recomputed with
// the same operations from the same inputs, so every bit equals the one-step
// kernel's (fused.cu).  Cells outside the grid hold values that no cell of the
// grid reads (the ghost rules replace every such neighbour).
//
// Fields and CPML memories (H and E) are read from one bank and written to the
// other; the launches of a call are split so that their number has the
// parity of its steps, which is where the caller expects the result.
//
// DFT samples and field recorders read single cells after every step: at its
// start a CTA lists the gather slots whose cell it owns, and after each step
// it writes those cells.  The slots come sorted by cell, with the first one of
// every 16 columns of a row, so that a CTA looks at its own only.  (When each
// CTA looked through all of them, and after every step once its list was full, a
// whole-plane monitor took 254 us per step at 400 x 400 and 4.7 ms at 1000 x
// 1000, now 11 and 60, in single steps 26 and 93; four lines of a 1000 x 1000
// plane 14.3, now 12.1.)  DFT samples go, slot by slot, to a ring of two
// halves; the next launch's first CTAs form the interpolated values and add the
// previous launch's steps to the arena (dft.cuh) beside the stepping CTAs, and
// one last launch adds the final ones.  Recorders write their record directly.
//
// Arithmetic follows beamz/simulation/kernels.py:731-877, 1217-1355 as in
// fused.cu (rounding contract in fdtd_common.cuh); sources at their three
// timings and PEC follow beamz/simulation/execute.py:374-541.

#include <algorithm>

#include "dft.cuh"

namespace fdtd {

namespace {

constexpr int kW = 64;                    // region columns
constexpr int kGroups = kW / 4;           // threads along x, four columns each
constexpr int kMaxT = 16;
constexpr int kEntryCap = 4096;           // listed gather slots per CTA (more: looked up after each step)
constexpr int kSlotLanes = 16;            // threads that share a row's gather slots
constexpr int kSmemTwo = 113 * 1024;      // dynamic shared memory that lets two CTAs share an SM
constexpr int kStatic = 2048;             // room for the static shared memory
constexpr int kSmemMax = kSmemTwo - kStatic;  // most dynamic shared memory of any plan

struct Geo2D {
  int T, TX, TY, rows, gx, gy;
  int nflush;             // leading CTAs that flush the previous launch's samples
  int flush_first, flush_count, flush_slot0;
  int slot0;              // this launch's first sample slot
  int step_offset;        // steps of the call before this launch
  int dft_cap, rec_cap;   // list capacities
  // dynamic shared memory, in floats from its start
  int o_coef, o_psi_hy, o_psi_hx, o_psi_ey, o_psi_ex, o_row, o_col, o_list;
};

struct Block2D {
  Step3D p;
  Geo2D g;
  DftDev d;
  SlotOrder slots;
  float* samples;
  const int* counter;
  int nsrc;
  SourceDev src[kMaxFusedSources];
  int timing[kMaxFusedSources];
  int nrec;
  RecorderDev rec[FDTD_MAX_RECORDERS];
};

// How a region of `len` coordinates from `lo` meets a term's slab: runs
// [lo0, lo0 + ln) and [hi0, hi0 + hn) in region coordinates.
struct SlabRuns {
  int lo0, ln, hi0, hn;
};
__host__ __device__ inline SlabRuns slab_runs(const CpmlTermDev& t, int lo, int len) {
  SlabRuns r{0, 0, 0, 0};
  const int a = lo > 0 ? lo : 0, b = (t.low < lo + len ? t.low : lo + len);
  if (b > a) {
    r.lo0 = a - lo;
    r.ln = b - a;
  }
  const int h0 = t.n_axis - t.high;
  const int c = h0 > lo ? h0 : lo, e = (t.n_axis < lo + len ? t.n_axis : lo + len);
  if (t.high > 0 && e > c) {
    r.hi0 = c - lo;
    r.hn = e - c;
  }
  return r;
}
__host__ __device__ inline int run_index(const SlabRuns& r, int x) {
  if (x >= r.lo0 && x < r.lo0 + r.ln) return x - r.lo0;
  if (x >= r.hi0 && x < r.hi0 + r.hn) return r.ln + x - r.hi0;
  return -1;
}

// psi <- b psi + a d, d' = d / kappa + psi (fdtd_common.cuh's cpml_correct).
__device__ __forceinline__ float corrected(const float4& c, float& psi, float d) {
  psi = c.y * psi + c.x * d;
  return d * c.z + psi;
}

struct V4 {
  float v[4];
};
__device__ __forceinline__ V4 ldv(const float* p) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  return {{a.x, a.y, a.z, a.w}};
}
__device__ __forceinline__ void stv(float* p, const V4& a) {
  *reinterpret_cast<float4*>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}

__device__ __forceinline__ void copy4(float* dst, const float* src, bool valid) {
  const unsigned at = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(at), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

// Column runs widened to whole groups of four region columns (the runs of a
// term's two slabs may then share a group: they merge).
__host__ __device__ inline SlabRuns group_runs(const SlabRuns& r) {
  SlabRuns o{0, 0, 0, 0};
  if (r.ln > 0) {
    o.lo0 = r.lo0 & ~3;
    o.ln = ((r.lo0 + r.ln + 3) & ~3) - o.lo0;
  }
  if (r.hn > 0) {
    o.hi0 = r.hi0 & ~3;
    int end = (r.hi0 + r.hn + 3) & ~3;
    if (o.ln > 0 && o.hi0 < o.lo0 + o.ln) o.hi0 = o.lo0 + o.ln;
    o.hn = end > o.hi0 ? end - o.hi0 : 0;
  }
  return o;
}

struct ListEntry {
  int src;    // shared-memory offset of the cell (-1: no cell, a zero is recorded)
  int dst;    // offset within a sample slot, or a record's value index
  float w;    // recorders: weight
  int which;  // recorders: recorder * 8 + component slot
};

// A tile's first own cell, and its number.
struct Tile {
  int i, j, n;
};

// f(position, shared-memory offset) for the slots sorted by cell whose cell of
// component c (table component `a`) lies in row `row` of the tile: the row's slots
// of the 16-column blocks that the tile meets, by kSlotLanes threads.
template <int Pol, class F>
__device__ __forceinline__ void own_slots(const Block2D& q, const SlotOrder& so, const int* cells, int total,
                                          const Tile& t, int a, int c, int row, int lane, F f) {
  constexpr int kC0 = Pol == 0 ? 2 : 5, kC1 = Pol == 0 ? 3 : 0;
  const Geo2D& g = q.g;
  const Dims d = component_dims_2d(c, Pol, q.p.Y, q.p.X);
  const int j = t.j + row;
  if (j >= d.y) return;
  const int blocks = (q.p.X + kSlotBlock) / kSlotBlock;
  const int* first = so.first + (a * (q.p.Y + 1) + j) * blocks;
  const int lo = max(__ldg(first + t.i / kSlotBlock), 0);
  const int hi = min(__ldg(first + min((t.i + g.TX + kSlotBlock - 1) / kSlotBlock, blocks)), so.n);
  const int from = j * d.x + t.i, width = min(g.TX, d.x - t.i);  // the row's own cells
  const int o = ((c == kC0 ? 0 : (c == kC1 ? 1 : 2)) * g.rows + row + g.T) * kW + g.T;
#pragma unroll 4
  for (int e = lo + lane; e < hi; e += kSlotLanes) {
    const int at = __ldg(so.order + e);
    if (at < 0 || at >= total) continue;
    const int x = __ldg(cells + at) - from;
    if (x >= 0 && x < width) f(at, o + x);
  }
}

// emit(cell, offset in a sample slot) for every DFT gather slot that the tile owns.
template <int Pol, class F>
__device__ __forceinline__ void own_samples(const Block2D& q, const Tile& t, int tid, int nthreads, F emit) {
  const int total = q.d.monitor_count * 6 * q.d.neighbors * q.d.max_points;
  for (int it = tid / kSlotLanes; it < 3 * q.g.TY; it += nthreads / kSlotLanes) {
    const int a = it / q.g.TY, c = Pol == 0 ? 2 + a : (a == 2 ? 5 : a);
    own_slots<Pol>(q, q.slots, q.d.indices, total, t, a, c, it - a * q.g.TY, tid % kSlotLanes,
                   [&](int at, int cell) { emit(cell, at); });
  }
}

// emit(cell, value, weight, which) for every value that the tile owns of recorder
// `only`'s (-1: every recorder's) sets that are neither whole components nor boxes.
// Tile 0 has the values without a cell (cell -1: a zero is recorded).
template <int Pol, class F>
__device__ __forceinline__ void own_values(const Block2D& q, int only, const Tile& t, int tid, int nthreads, F emit) {
  for (int n = 0; n < q.nrec; ++n) {
    if (only >= 0 && n != only) continue;
    const RecorderDev& rec = q.rec[n];
    for (int v = 0; v < rec.ncomp; ++v) {
      if (rec.slots[v] == 0 || rec.box[v].ny > 0) continue;
      const int V = static_cast<int>(rec.start[v + 1] - rec.start[v]);
      const SlotOrder& so = rec.order[v];
      for (int row = tid / kSlotLanes; row < q.g.TY; row += nthreads / kSlotLanes)
        own_slots<Pol>(q, so, rec.idx[v], V, t, 0, rec.comp[v], row, tid % kSlotLanes,
                       [&](int at, int cell) { emit(cell, at, rec.w[v][at], n * 8 + v); });
      if (t.n != 0) continue;
      const int blocks = (q.p.X + kSlotBlock) / kSlotBlock;
      for (int e = max(so.first[(q.p.Y + 1) * blocks], 0) + tid; e < V; e += nthreads) {
        const int at = so.order[e];
        if (at >= 0 && at < V) emit(-1, at, 0.0f, n * 8 + v);
      }
    }
  }
}

__device__ __forceinline__ void record_value(const RecorderDev& rec, const ListEntry& e, int at, const float* sm) {
  const int v = e.which & 7;
  const int64_t V = rec.start[v + 1] - rec.start[v];
  const float x = e.src >= 0 ? 0.0f + sm[e.src] * e.w : 0.0f;
  rec.values[v][at * V + e.dst] = x * rec.sign[v];
}

// A step's samples and values of a tile that owns more of them than its list holds;
// out of line, so that the steps' loop stays short.
template <int Pol>
__device__ __noinline__ void sample_unlisted(const Block2D& q, const Tile t, int tid, int nthreads, float* out,
                                             const float* sm) {
  own_samples<Pol>(q, t, tid, nthreads, [&](int src, int dst) { out[dst] = sm[src]; });
}
template <int Pol>
__device__ __noinline__ void record_unlisted(const Block2D& q, int n, const Tile t, int tid, int nthreads, int at,
                                             const float* sm) {
  own_values<Pol>(q, n, t, tid, nthreads, [&](int src, int dst, float w, int which) {
    record_value(q.rec[n], ListEntry{src, dst, w, which}, at, sm);
  });
}

// Pol 0: TM (Ez, Hx, Hy); 1: TE (Hz, Ex, Ey).  Site: every coefficient is
// staged per cell; else only the E sources are (E decay and H uniform).
// kThreads, PerSm: the launch shape (launch_shape below).
template <int Pol, bool Cpml, bool Site, bool Metric, int kThreads, int PerSm>
__global__ void __launch_bounds__(kThreads, PerSm) block2d_kernel(const __grid_constant__ Block2D q) {
  constexpr int kRows = kThreads / kGroups;  // rows in flight
  extern __shared__ __align__(16) float sm[];
  const Step3D& p = q.p;
  const Geo2D& g = q.g;
  const int tid = threadIdx.x;
  // Components: F0 is the single one (TM: Ez, TE: Hz), F1 its partner in y
  // (Hx / Ex), F2 its partner in x (Hy / Ey).
  constexpr int kC0 = Pol == 0 ? 2 : 5, kC1 = Pol == 0 ? 3 : 0, kC2 = Pol == 0 ? 4 : 1;
  if (static_cast<int>(blockIdx.x) < g.nflush) {
    const int chunks = (q.d.max_points + kThreads - 1) / kThreads;
    const int chunk = blockIdx.x % chunks, mc = blockIdx.x / chunks;
    const int m = mc / 3, a = mc % 3;
    dft_flush_body<true>(q.d, *reinterpret_cast<FlushShared*>(sm), q.samples, q.counter, g.flush_first, g.flush_slot0,
                         g.flush_count, m, a == 0 ? kC0 : (a == 1 ? kC1 : kC2), chunk * kThreads, a == 0 && chunk == 0,
                         tid, kThreads);
    return;
  }
  const int tile = blockIdx.x - g.nflush;
  const int tx = tile % g.gx, ty = tile / g.gx;
  const int T = g.T, H = g.rows;
  const int own_i = tx * g.TX, own_j = ty * g.TY;
  const Tile own{own_i, own_j, tile};
  const int i0 = own_i - T, j0 = own_j - T;  // region origin
  const int Y = p.Y, X = p.X;
  // Component extents (y, x).
  const int y0n = Pol == 0 ? Y + 1 : Y, x0n = Pol == 0 ? X + 1 : X;  // F0
  const int y1n = Pol == 0 ? Y : Y + 1, x1n = Pol == 0 ? X + 1 : X;  // F1
  const int y2n = Pol == 0 ? Y + 1 : Y, x2n = Pol == 0 ? X : X + 1;  // F2
  const int plane = H * kW;
  float* F0 = sm;
  float* F1 = sm + plane;
  float* F2 = sm + 2 * plane;
  float* coef = sm + g.o_coef;
  // CPML terms: y terms act on F1 (TM: Hx from ht[0]; TE: Ex from et[0]) and on
  // F0 (TM: Ez from et[5]; TE: Hz from ht[5]); x terms on F2 (TM: Hy ht[3];
  // TE: Ey et[3]) and F0 (TM: Ez et[4]; TE: Hz ht[4]).
  const CpmlTermDev& t1 = Pol == 0 ? p.ht[0] : p.et[0];   // F1, y
  const CpmlTermDev& t2 = Pol == 0 ? p.ht[3] : p.et[3];   // F2, x
  const CpmlTermDev& t0y = Pol == 0 ? p.et[5] : p.ht[5];  // F0, y
  const CpmlTermDev& t0x = Pol == 0 ? p.et[4] : p.ht[4];  // F0, x
  float* psi1 = sm + g.o_psi_hy;
  float* psi2 = sm + g.o_psi_hx;
  float* psi0y = sm + g.o_psi_ey;
  float* psi0x = sm + g.o_psi_ex;
  // Per-row and per-column CPML coefficients (a, b, 1/kappa); .w of a row its
  // compact psi row, of a column 0 inside the slab (-1: outside).
  float4* row1 = reinterpret_cast<float4*>(sm + g.o_row);
  float4* row0 = row1 + H;
  float4* col2 = reinterpret_cast<float4*>(sm + g.o_col);
  float4* col0 = col2 + kW;
  SlabRuns r1{}, r0{}, c2{}, c0{};
  if constexpr (Cpml) {
    r1 = slab_runs(t1, j0, H);
    r0 = slab_runs(t0y, j0, H);
    c2 = group_runs(slab_runs(t2, i0, kW));
    c0 = group_runs(slab_runs(t0x, i0, kW));
  }
  const int n2 = c2.ln + c2.hn, n0 = c0.ln + c0.hn;  // compact psi columns (whole groups)
  auto rows_of = [&](const SlabRuns& r, int e) { return e < r.ln ? r.lo0 + e : r.hi0 + e - r.ln; };

  // ---- load: every copy goes out before anything is waited for -------------------
  const float* in0 = Pol == 0 ? p.ein[2] : p.hin[2];
  const float* in1 = Pol == 0 ? p.hin[0] : p.ein[0];
  const float* in2 = Pol == 0 ? p.hin[1] : p.ein[1];
  {
    const int col = tid & (kW - 1), ry = tid / kW, i = i0 + col;
    auto load_plane = [&](float* dst, const float* src, int yn, int xn) {
      const bool iok = i >= 0 && i < xn;
#pragma unroll 4
      for (int r = ry; r < H; r += kThreads / kW) {
        const int j = j0 + r;
        const bool ok = iok && j >= 0 && j < yn;
        copy4(dst + r * kW + col, src + (ok ? j * xn + i : 0), ok);
      }
    };
    auto fill_plane = [&](float* dst, const float* src, bool full, int yn, int xn) {
      if (full) {
        load_plane(dst, src, yn, xn);
      } else {
        const float v = src[0];
        for (int r = ry; r < H; r += kThreads / kW) dst[r * kW + col] = v;
      }
    };
    load_plane(F0, in0, y0n, x0n);
    load_plane(F1, in1, y1n, x1n);
    load_plane(F2, in2, y2n, x2n);
    if constexpr (Site) {
      auto both = [&](int f, int c, int yn, int xn) {
        const bool e = c < 3;
        const int k = e ? c : c - 3;
        fill_plane(coef + 2 * f * plane, e ? p.em.decay[k] : p.hm.decay[k],
                   e ? p.em.decay_full[k] : p.hm.decay_full[k], yn, xn);
        fill_plane(coef + (2 * f + 1) * plane, e ? p.em.source[k] : p.hm.source[k],
                   e ? p.em.source_full[k] : p.hm.source_full[k], yn, xn);
      };
      both(0, kC0, y0n, x0n);
      both(1, kC1, y1n, x1n);
      both(2, kC2, y2n, x2n);
    } else if constexpr (Pol == 0) {
      fill_plane(coef, p.em.source[2], p.em.source_full[2], y0n, x0n);
    } else {
      fill_plane(coef, p.em.source[0], p.em.source_full[0], y1n, x1n);
      fill_plane(coef + plane, p.em.source[1], p.em.source_full[1], y2n, x2n);
    }
    if constexpr (Cpml) {
      auto load_y = [&](const CpmlTermDev& t, const SlabRuns& r, float* psi, int xn) {
        const bool ok = i >= 0 && i < xn;
        for (int e = ry; e < r.ln + r.hn; e += kThreads / kW) {
          const int slot = cpml_slot(t, j0 + rows_of(r, e));
          copy4(psi + e * kW + col, t.psi_in + (ok ? slot * t.pdx + i : 0), ok);
        }
      };
      auto load_x = [&](const CpmlTermDev& t, const SlabRuns& r, float* psi, int n, int yn) {
        for (int e = tid; e < H * n; e += kThreads) {
          const int rr = e / n, j = j0 + rr, at = i0 + rows_of(r, e - rr * n);
          const int slot = at >= 0 && at < t.n_axis ? cpml_slot(t, at) : -1;
          const bool ok = slot >= 0 && j >= 0 && j < yn;
          copy4(psi + e, t.psi_in + (ok ? j * t.pdx + slot : 0), ok);
        }
      };
      if (r1.ln + r1.hn) load_y(t1, r1, psi1, x1n);
      if (r0.ln + r0.hn) load_y(t0y, r0, psi0y, x0n);
      if (n2) load_x(t2, c2, psi2, n2, y2n);
      if (n0) load_x(t0x, c0, psi0x, n0, y0n);
    }
  }
  __shared__ float amp[kMaxFusedSources][kMaxT];
  __shared__ int live[kMaxFusedSources];  // sources whose box meets this region
  __shared__ int nlist, nrlist;
  if (tid == 0) nlist = nrlist = 0;
  const int step0 = q.counter[0] + g.step_offset;
  for (int e = tid; e < q.nsrc * kMaxT; e += kThreads) {
    const int s = e / kMaxT, t = e % kMaxT;
    if (t < T) amp[s][t] = source_amplitude(q.src[s], step0 + t);
  }
  if (tid < q.nsrc) {
    const SourceDev& s = q.src[tid];
    live[tid] = s.y0 < j0 + H && s.y0 + s.ey > j0 && s.x0 < i0 + kW && s.x0 + s.ex > i0;
  }
  if constexpr (Cpml) {
    for (int e = tid; e < 2 * H + 2 * kW; e += kThreads) {
      const bool is_row = e < 2 * H;
      const int w = is_row ? (e >= H) : (e - 2 * H >= kW), x = is_row ? e - w * H : e - 2 * H - w * kW;
      const CpmlTermDev& t = is_row ? (w ? t0y : t1) : (w ? t0x : t2);
      const int at = (is_row ? j0 : i0) + x;
      const int slot = at >= 0 && at < t.n_axis ? cpml_slot(t, at) : -1;
      float4 v = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
      if (slot >= 0) v = make_float4(t.a[slot], t.b[slot], t.k[slot], __int_as_float(is_row ? run_index(w ? r0 : r1, x) : 0));
      (is_row ? (w ? row0 : row1) : (w ? col0 : col2))[x] = v;
    }
  }
  float dec0 = 1.0f, dec1 = 1.0f, dec2 = 1.0f, us0 = 0.0f, us1 = 0.0f, us2 = 0.0f;
  if constexpr (!Site && Pol == 0) {
    dec0 = p.em.decay[2][0];
    dec1 = p.hm.decay[0][0];
    dec2 = p.hm.decay[1][0];
    us1 = p.hm.source[0][0];
    us2 = p.hm.source[1][0];
  }
  if constexpr (!Site && Pol == 1) {
    dec0 = p.hm.decay[2][0];
    dec1 = p.em.decay[0][0];
    dec2 = p.em.decay[1][0];
    us0 = p.hm.source[2][0];
  }
  __syncthreads();  // list counters
  // ---- the cells that monitors and recorders read ------------------------------
  auto plane_of = [&](int c, int* yn, int* xn) {
    const int f = c == kC0 ? 0 : (c == kC1 ? 1 : 2);
    *yn = f == 0 ? y0n : (f == 1 ? y1n : y2n);
    *xn = f == 0 ? x0n : (f == 1 ? x1n : x2n);
    return f * plane;
  };
  ListEntry* rlist = reinterpret_cast<ListEntry*>(sm + g.o_list);
  int2* list = reinterpret_cast<int2*>(rlist + g.rec_cap);
  if (q.samples != nullptr)
    own_samples<Pol>(q, own, tid, kThreads, [&](int src, int dst) {
      const int n = atomicAdd(&nlist, 1);
      if (n < g.dft_cap) list[n] = make_int2(src, dst);
    });
  if (g.rec_cap)
    own_values<Pol>(q, -1, own, tid, kThreads, [&](int src, int dst, float w, int which) {
      const int n = atomicAdd(&nrlist, 1);
      if (n < g.rec_cap) rlist[n] = ListEntry{src, dst, w, which};
    });
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  const int entries = nlist, rentries = nrlist;
  bool any_pre = false, any_h = false, any_e = false;
  for (int s = 0; s < q.nsrc; ++s)
    if (live[s]) {
      any_pre |= q.timing[s] == FDTD_TIMING_PRE_E;
      any_h |= q.timing[s] == FDTD_TIMING_H;
      any_e |= q.timing[s] == FDTD_TIMING_E;
    }

  const int grp = tid & (kGroups - 1), ry = tid / kGroups;
  const int c4 = 4 * grp, i = i0 + c4;  // this thread's first column
  const unsigned half = 0xffffu << (tid & 16);  // the half warp of this thread's row
  const bool wy0 = wall(p.metallic, 1, false), wy1 = wall(p.metallic, 1, true);
  const bool wx0 = wall(p.metallic, 2, false), wx1 = wall(p.metallic, 2, true);
  // This thread's columns x = 0 and x = X (their position among its four, else
  // outside 0..3).
  const int at0 = -i, atX = X - i;
  const bool edge = (at0 >= 0 && at0 < 4) || (atX >= 0 && atX < 4);
  // x terms: the group's compact psi columns and which of its columns lie in
  // the slab.
  int g2 = -1, g0 = -1, m2 = 0, m0 = 0;
  if constexpr (Cpml) {
    g2 = run_index(c2, c4);
    g0 = run_index(c0, c4);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m2 |= (__float_as_int(col2[c4 + k].w) >= 0) << k;
      m0 |= (__float_as_int(col0[c4 + k].w) >= 0) << k;
    }
    if (m2 == 0) g2 = -1;
    if (m0 == 0) g0 = -1;
  }
  // Derivatives of four cells: forward (H) and backward (E), along x at columns
  // i.. and along y at row j.
  auto scale_x = [&](V4& d, bool fwd) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (Metric) d.v[k] = d.v[k] * (fwd ? p.metric_h[2][clampi(i + k, X - 1)] : p.metric_e[2][clampi(i + k, X)]);
      else d.v[k] = div_rn(d.v[k], p.div_bs, p.div_rs);
    }
  };
  auto scale_y = [&](V4& d, bool fwd, int j) {
    float m = 1.0f;
    if constexpr (Metric) m = fwd ? p.metric_h[1][clampi(j, Y - 1)] : p.metric_e[1][clampi(j, Y)];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (Metric) d.v[k] = d.v[k] * m;
      else d.v[k] = div_rn(d.v[k], p.div_bs, p.div_rs);
    }
  };
  // f(x + 1) - f(x) and f(y + 1) - f(y).
  auto fwd_x = [&](const V4& f) {
    const float n = __shfl_down_sync(half, f.v[0], 1, kGroups);
    V4 d{{f.v[1] - f.v[0], f.v[2] - f.v[1], f.v[3] - f.v[2], n - f.v[3]}};
    scale_x(d, true);
    return d;
  };
  auto fwd_y = [&](const V4& f, const V4& up, int j) {
    V4 d;
#pragma unroll
    for (int k = 0; k < 4; ++k) d.v[k] = up.v[k] - f.v[k];
    scale_y(d, true, j);
    return d;
  };
  // Ghost-padded backward differences (beamz/lattice.py:523-551): zero beyond a
  // metallic wall, else a copy of the edge sample (the difference vanishes).
  auto back_x = [&](const V4& f) {
    const float b = __shfl_up_sync(half, f.v[3], 1, kGroups);
    V4 d{{f.v[0] - b, f.v[1] - f.v[0], f.v[2] - f.v[1], f.v[3] - f.v[2]}};
    if (edge) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k == at0) d.v[k] = wx0 ? f.v[k] - 0.0f : 0.0f;
        if (k == atX) d.v[k] = wx1 ? 0.0f - (k ? f.v[k ? k - 1 : 0] : b) : 0.0f;
      }
    }
    scale_x(d, false);
    return d;
  };
  auto back_y = [&](const V4& f, const V4& below, int j) {
    V4 d;
#pragma unroll
    for (int k = 0; k < 4; ++k) d.v[k] = f.v[k] - below.v[k];
    if (j == 0 || j == Y) {
      const bool w = j == 0 ? wy0 : wy1;
#pragma unroll
      for (int k = 0; k < 4; ++k) d.v[k] = w ? (j == 0 ? f.v[k] - 0.0f : 0.0f - below.v[k]) : 0.0f;
    }
    scale_y(d, false, j);
    return d;
  };
  // CPML corrections of four cells.
  auto cpml_y = [&](V4& d, const float4* rows, float* psi, int r) {
    if constexpr (Cpml) {
      const float4 c = rows[r];
      const int s = __float_as_int(c.w);
      if (s < 0) return;
      float* at = psi + s * kW + c4;
      V4 v = ldv(at);
#pragma unroll
      for (int k = 0; k < 4; ++k) d.v[k] = corrected(c, v.v[k], d.v[k]);
      stv(at, v);
    }
  };
  auto cpml_x = [&](V4& d, const float4* cols, float* psi, int n, int gi, int mask, int r) {
    if constexpr (Cpml) {
      if (gi < 0) return;
      float* at = psi + r * n + gi;
      V4 v = ldv(at);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (mask & (1 << k)) d.v[k] = corrected(cols[c4 + k], v.v[k], d.v[k]);
      stv(at, v);
    }
  };
  // Decay and source of field f at the four cells from region cell o.
  auto dec_of = [&](int f, int o) -> V4 {
    if constexpr (Site) return ldv(coef + 2 * f * plane + o);
    const float v = f == 0 ? dec0 : (f == 1 ? dec1 : dec2);
    return {{v, v, v, v}};
  };
  auto src_of = [&](int f, int o) -> V4 {
    if constexpr (Site) return ldv(coef + (2 * f + 1) * plane + o);
    if (Pol == 0 && f == 0) return ldv(coef + o);
    if (Pol == 1 && f > 0) return ldv(coef + (f - 1) * plane + o);
    const float v = f == 0 ? us0 : (f == 1 ? us1 : us2);
    return {{v, v, v, v}};
  };
  // Every source of `timing` on component c covering row j, in order.
  auto inject = [&](int timing, int c, int j, V4& v, int t) {
#pragma unroll 1
    for (int s = 0; s < q.nsrc; ++s) {
      if (!live[s] || q.timing[s] != timing || q.src[s].component != c) continue;
      const SourceDev& sr = q.src[s];
      const int y = j - sr.y0;
      if (y < 0 || y >= sr.ey) continue;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int x = i + k - sr.x0;
        if (x >= 0 && x < sr.ex) v.v[k] = v.v[k] + sr.coeff[y * sr.ex + x] * amp[s][t];
      }
    }
  };
  // PEC on the metallic x walls (bit 0: x = 0, bit 1: x = X).
  auto zero_x = [&](V4& v) {
    if (!edge) return;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if ((wx0 && k == at0) || (wx1 && k == atX)) v.v[k] = 0.0f;
  };
  auto zero_y = [&](V4& v, int j) {
    if ((wy0 && j == 0) || (wy1 && j == Y)) v = V4{{0.f, 0.f, 0.f, 0.f}};
  };

  for (int t = 0; t < T; ++t) {
    const int rem = T - 1 - t;
    const int e_lo = T - rem, e_hi = T + g.TY + rem;  // E rows that later steps need
    if (any_pre) {
      for (int r = ry; r < H; r += kRows) {
        const int j = j0 + r, o = r * kW + c4;
        if constexpr (Pol == 0) {
          V4 v = ldv(F0 + o);
          inject(FDTD_TIMING_PRE_E, kC0, j, v, t);
          stv(F0 + o, v);
        } else {
          V4 v = ldv(F1 + o), w = ldv(F2 + o);
          inject(FDTD_TIMING_PRE_E, kC1, j, v, t);
          inject(FDTD_TIMING_PRE_E, kC2, j, w, t);
          stv(F1 + o, v);
          stv(F2 + o, w);
        }
      }
      __syncthreads();
    }
    // ---- H -------------------------------------------------------------------
    // A warp covers two rows; both run when either is needed.
    for (int r = ry; r < H; r += kRows) {
      if ((r | 1) < e_lo - 1 || (r & ~1) >= e_hi) continue;
      const int j = j0 + r, o = r * kW + c4, up = r + 1 < H ? o + kW : o;
      if constexpr (Pol == 0) {
        const V4 ez = ldv(F0 + o);
        V4 d0 = fwd_y(ez, ldv(F0 + up), j);  // Hx: dEz/dy
        V4 d1 = fwd_x(ez);                   // Hy: -dEz/dx
        cpml_y(d0, row1, psi1, r);
        cpml_x(d1, col2, psi2, n2, g2, m2, r);
        V4 hx = ldv(F1 + o), hy = ldv(F2 + o);
        const V4 ax = dec_of(1, o), bx = src_of(1, o), ay = dec_of(2, o), by = src_of(2, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          hx.v[k] = ax.v[k] * hx.v[k] - bx.v[k] * (d0.v[k] - 0.0f);
          hy.v[k] = ay.v[k] * hy.v[k] - by.v[k] * (0.0f - d1.v[k]);
        }
        if (any_h) {
          inject(FDTD_TIMING_H, kC1, j, hx, t);
          inject(FDTD_TIMING_H, kC2, j, hy, t);
        }
        zero_x(hx);
        zero_y(hy, j);
        stv(F1 + o, hx);
        stv(F2 + o, hy);
      } else {
        const V4 ex = ldv(F1 + o), ey = ldv(F2 + o);
        V4 d0 = fwd_x(ey), d1 = fwd_y(ex, ldv(F1 + up), j);  // Hz: dEy/dx - dEx/dy
        cpml_x(d0, col0, psi0x, n0, g0, m0, r);
        cpml_y(d1, row0, psi0y, r);
        V4 hz = ldv(F0 + o);
        const V4 a = dec_of(0, o), b = src_of(0, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) hz.v[k] = a.v[k] * hz.v[k] - b.v[k] * (d0.v[k] - d1.v[k]);
        if (any_h) inject(FDTD_TIMING_H, kC0, j, hz, t);
        stv(F0 + o, hz);
      }
    }
    __syncthreads();
    // ---- E -------------------------------------------------------------------
    for (int r = ry; r < H; r += kRows) {
      if ((r | 1) < e_lo || (r & ~1) >= e_hi) continue;
      const int j = j0 + r, o = r * kW + c4, down = r > 0 ? o - kW : o;
      if constexpr (Pol == 0) {  // Ez: dHy/dx - dHx/dy
        V4 d0 = back_x(ldv(F2 + o)), d1 = back_y(ldv(F1 + o), ldv(F1 + down), j);
        cpml_x(d0, col0, psi0x, n0, g0, m0, r);
        cpml_y(d1, row0, psi0y, r);
        V4 e = ldv(F0 + o);
        const V4 a = dec_of(0, o), b = src_of(0, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) e.v[k] = a.v[k] * e.v[k] + b.v[k] * (d0.v[k] - d1.v[k]);
        if (any_e) inject(FDTD_TIMING_E, kC0, j, e, t);
        zero_x(e);
        zero_y(e, j);
        stv(F0 + o, e);
      } else {
        const V4 hz = ldv(F0 + o);
        V4 d0 = back_y(hz, ldv(F0 + down), j), d1 = back_x(hz);  // Ex: dHz/dy; Ey: -dHz/dx
        cpml_y(d0, row1, psi1, r);
        cpml_x(d1, col2, psi2, n2, g2, m2, r);
        V4 ex = ldv(F1 + o), ey = ldv(F2 + o);
        const V4 ax = dec_of(1, o), bx = src_of(1, o), ay = dec_of(2, o), by = src_of(2, o);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          ex.v[k] = ax.v[k] * ex.v[k] + bx.v[k] * (d0.v[k] - 0.0f);
          ey.v[k] = ay.v[k] * ey.v[k] + by.v[k] * (0.0f - d1.v[k]);
        }
        if (any_e) {
          inject(FDTD_TIMING_E, kC1, j, ex, t);
          inject(FDTD_TIMING_E, kC2, j, ey, t);
        }
        zero_y(ex, j);
        zero_x(ey);
        stv(F1 + o, ex);
        stv(F2 + o, ey);
      }
    }
    __syncthreads();
    // ---- samples and records -----------------------------------------------------
    if (entries) {
      const int64_t stride = static_cast<int64_t>(q.d.monitor_count) * 6 * q.d.neighbors * q.d.max_points;
      float* out = q.samples + (g.slot0 + t) * stride;
      if (entries <= g.dft_cap) {
        for (int e = tid; e < entries; e += kThreads) out[list[e].y] = sm[list[e].x];
      } else {
        sample_unlisted<Pol>(q, own, tid, kThreads, out, sm);
      }
    }
    for (int n = 0; n < q.nrec; ++n) {
      const RecorderDev& rec = q.rec[n];
      const int s0 = q.counter[0], step = step0 + t;  // s0: the call's first step
      if ((step + 1) % rec.interval != 0) continue;
      const int at = rec.count[s0 & 1] + step / rec.interval - s0 / rec.interval;
      if (at >= rec.capacity) continue;
      if (tile == 0 && tid == 0) {
        rec.steps[at] = step + 1;
        rec.times[at] = rec.step_time[step < rec.step_time_len ? step : rec.step_time_len - 1];
      }
      if (rentries > g.rec_cap) {
        record_unlisted<Pol>(q, n, own, tid, kThreads, at, sm);
      } else {
        for (int e = tid; e < rentries; e += kThreads)
          if (rlist[e].which >> 3 == n) record_value(rec, rlist[e], at, sm);
      }
      for (int v = 0; v < rec.ncomp; ++v) {  // whole components and boxes: the tile's part of them
        int yn, xn, lo_y = 0, lo_x = 0;
        const float* f = sm + plane_of(rec.comp[v], &yn, &xn);
        int by = yn, bx = xn;
        if (rec.slots[v] != 0) {
          lo_y = rec.box[v].y0;
          lo_x = rec.box[v].x0;
          by = rec.box[v].ny;
          bx = rec.box[v].nx;
        }
        const bool plain = rec.slots[v] == 0;
        const int64_t V = rec.start[v + 1] - rec.start[v];
        float* out = rec.values[v] + at * V;
        const int j_lo = max(own_j, lo_y), j_hi = min(own_j + g.TY, lo_y + by);
        const int col = tid & (kW - 1), x = i0 + col;
        if (col < T || col >= T + g.TX || x < lo_x || x >= lo_x + bx) continue;
        for (int j = j_lo + tid / kW; j < j_hi; j += kThreads / kW) {
          const float val = f[(j - j0) * kW + col];
          out[(j - lo_y) * bx + x - lo_x] = (plain ? val : 0.0f + val * 1.0f) * rec.sign[v];
        }
      }
    }
    if (t + 1 < T && (entries || q.nrec)) __syncthreads();  // before the next step overwrites the cells
  }

  // ---- store the tile ------------------------------------------------------------
  float* out0 = Pol == 0 ? p.eout[2] : p.hout[2];
  float* out1 = Pol == 0 ? p.hout[0] : p.eout[0];
  float* out2 = Pol == 0 ? p.hout[1] : p.eout[1];
  const int col = tid & (kW - 1), x = i0 + col;
  const bool mine = col >= T && col < T + g.TX;
  if (mine) {
#pragma unroll 4
    for (int r = T + tid / kW; r < T + g.TY; r += kThreads / kW) {
      const int j = j0 + r, o = r * kW + col;
      if (j < y0n && x < x0n) out0[j * x0n + x] = F0[o];
      if (j < y1n && x < x1n) out1[j * x1n + x] = F1[o];
      if (j < y2n && x < x2n) out2[j * x2n + x] = F2[o];
    }
  }
  if constexpr (Cpml) {
    auto store_y = [&](const CpmlTermDev& t, const SlabRuns& r, const float* psi, int xn) {
      for (int e = tid / kW; e < r.ln + r.hn; e += kThreads / kW) {
        const int rr = rows_of(r, e);
        if (mine && x < xn && rr >= T && rr < T + g.TY) t.psi_out[cpml_slot(t, j0 + rr) * t.pdx + x] = psi[e * kW + col];
      }
    };
    auto store_x = [&](const CpmlTermDev& t, const SlabRuns& r, const float* psi, int n, int yn) {
      for (int e = tid; e < g.TY * n; e += kThreads) {
        const int rr = T + e / n, cx = e % n, cl = rows_of(r, cx), j = j0 + rr, at = i0 + cl;
        if (j >= yn || cl < T || cl >= T + g.TX || at >= t.n_axis) continue;
        const int slot = cpml_slot(t, at);
        if (slot >= 0) t.psi_out[j * t.pdx + slot] = psi[rr * n + cx];
      }
    };
    store_y(t1, r1, psi1, x1n);
    store_y(t0y, r0, psi0y, x0n);
    if (n2) store_x(t2, c2, psi2, n2, y2n);
    if (n0) store_x(t0x, c0, psi0x, n0, y0n);
  }
}

__global__ void __launch_bounds__(256) flush_raw_kernel(DftDev d, const float* samples, const int* counter, int first,
                                                        int slot0, int count, int pol) {
  __shared__ FlushShared sh;
  const int m = blockIdx.y / 3, a = blockIdx.y % 3;
  const int c = pol == 0 ? (a == 0 ? 2 : 2 + a) : (a == 0 ? 5 : a - 1);
  dft_flush_body<true>(d, sh, samples, counter, first, slot0, count, m, c, blockIdx.x * blockDim.x,
                       a == 0 && blockIdx.x == 0, threadIdx.x, blockDim.x);
}

// The end of a call: the recorders' counts and the step counter.
__global__ void finish_kernel(int* counter, int nsteps, int nrec, RecorderDev r0, RecorderDev r1, RecorderDev r2,
                              RecorderDev r3) {
  const int s0 = counter[0], s1 = s0 + nsteps;
  auto count = [&](const RecorderDev& r) {
    const int n = r.count[s0 & 1] + s1 / r.interval - s0 / r.interval;
    const int to = n < r.capacity ? n : r.capacity;
    r.count[0] = to;
    r.count[1] = to;
  };
  if (nrec > 0) count(r0);
  if (nrec > 1) count(r1);
  if (nrec > 2) count(r2);
  if (nrec > 3) count(r3);
  counter[0] = s1;
}

struct Plan2D {
  Geo2D g;
  size_t smem;
};

int slab_max(const CpmlTermDev& t, int tiles, int own, int T, int len, bool groups) {
  int most = 0;
  for (int b = 0; b < tiles; ++b) {
    SlabRuns r = slab_runs(t, b * own - T, len);
    if (groups) r = group_runs(r);
    most = std::max(most, r.ln + r.hn);
  }
  return most;
}

// Tile shape for T steps per launch: 64 - 2T own columns, and own rows so that
// one tile per SM covers the grid, or, where such a tile would not leave an SM
// room for a second CTA, as few whole waves of smaller ones as do.
bool plan_tiles(const Block2D& q, int pol, bool site, int T, int sms, Plan2D* out) {
  const Step3D& p = q.p;
  Geo2D g{};
  g.T = T;
  g.TX = kW - 2 * T;
  g.gx = (p.X + 1 + g.TX - 1) / g.TX;
  const int planes = 3 + (site ? 6 : (pol == 0 ? 1 : 2));
  const CpmlTermDev& t1 = pol == 0 ? p.ht[0] : p.et[0];
  const CpmlTermDev& t2 = pol == 0 ? p.ht[3] : p.et[3];
  const CpmlTermDev& t0y = pol == 0 ? p.et[5] : p.ht[5];
  const CpmlTermDev& t0x = pol == 0 ? p.et[4] : p.ht[4];
  const int c2 = p.cpml ? slab_max(t2, g.gx, g.TX, T, kW, true) : 0;
  const int c0 = p.cpml ? slab_max(t0x, g.gx, g.TX, T, kW, true) : 0;
  bool lists = false;
  for (int n = 0; n < q.nrec; ++n)
    for (int v = 0; v < q.rec[n].ncomp; ++v) lists |= q.rec[n].slots[v] != 0 && q.rec[n].box[v].ny == 0;
  for (int waves = 1; waves <= 4096; ++waves) {
    const int per = waves * sms / g.gx;  // tile rows in `waves` waves
    if (per < 1) continue;
    g.TY = std::max(8, (p.Y + 1 + per - 1) / per);
    g.gy = (p.Y + 1 + g.TY - 1) / g.TY;
    g.rows = g.TY + 2 * T;
    const int r1 = p.cpml ? slab_max(t1, g.gy, g.TY, T, g.rows, false) : 0;
    const int r0 = p.cpml ? slab_max(t0y, g.gy, g.TY, T, g.rows, false) : 0;
    int at = planes * g.rows * kW;
    g.o_coef = 3 * g.rows * kW;
    auto take = [&](int n) {
      const int o = at;
      at += (n + 3) & ~3;
      return o;
    };
    g.o_row = take(p.cpml ? 8 * g.rows : 0);
    g.o_col = take(p.cpml ? 8 * kW : 0);
    g.o_psi_hy = take(r1 * kW);
    g.o_psi_ey = take(r0 * kW);
    g.o_psi_hx = take(c2 * g.rows);
    g.o_psi_ex = take(c0 * g.rows);
    g.rec_cap = lists ? std::min(kEntryCap, g.TY * g.TX) : 0;
    g.dft_cap = q.samples ? std::min(kEntryCap, g.TY * g.TX) : 0;
    g.o_list = take(4 * g.rec_cap + 2 * g.dft_cap);
    const size_t bytes = std::max(static_cast<size_t>(at) * 4, sizeof(FlushShared));
    if (bytes > kSmemMax) {
      if (g.TY == 8) return false;
      continue;
    }
    out->g = g;
    out->smem = bytes;
    return true;
  }
  return false;
}

template <int Pol, bool Cpml, bool Site, bool Metric, int Threads, int PerSm>
cudaError_t launch_s(cudaStream_t s, const Block2D& q, int ctas, size_t smem) {
  auto kern = block2d_kernel<Pol, Cpml, Site, Metric, Threads, PerSm>;
  // The limit belongs to the function, not to the launch: every thread sets the
  // same one, so that none lowers it between another's setting and its launch.
  const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
  if (err != cudaSuccess) return err;
  kern<<<ctas, Threads, smem, s>>>(q);
  return cudaPeekAtLastError();
}

// Threads of a CTA: 512, or 768 for tiles of one wave that are taller than the 32
// rows that 512 threads have in flight.
int launch_threads(const Geo2D& g, int sms) { return g.gx * g.gy <= sms && g.rows > 512 / kGroups ? 768 : 512; }

// Grids of one wave have an SM to themselves per tile: the steps are then bound
// by a tile's own instruction chain, and up to 128 (80) registers a thread shorten
// it; larger grids run two tiles per SM (us per step with one line monitor, 512
// threads two per SM / 512 one per SM / 768: 200 x 200 TM 3.81 / 3.29 / 3.58,
// 400 x 400 5.13 / 4.34 / 4.08, 83 x 117 TE 3.88 / 3.36 / 3.56, 1000 x 1000 12.4 /
// 11.8 / 13.0, 3000 x 3000 67 / 81 / 84).
template <int Pol, bool Cpml, bool Site, bool Metric>
cudaError_t launch_t(cudaStream_t s, const Block2D& q, int sms, int ctas, size_t smem) {
  if (q.g.gx * q.g.gy > sms) return launch_s<Pol, Cpml, Site, Metric, 512, 2>(s, q, ctas, smem);
  if (launch_threads(q.g, sms) == 768) return launch_s<Pol, Cpml, Site, Metric, 768, 1>(s, q, ctas, smem);
  return launch_s<Pol, Cpml, Site, Metric, 512, 1>(s, q, ctas, smem);
}

template <int Pol>
cudaError_t launch_pol(cudaStream_t s, const Block2D& q, bool site, int sms, int ctas, size_t smem) {
  const bool metric = has_metric(q.p);
  if (q.p.cpml) {
    if (metric)
      return site ? launch_t<Pol, true, true, true>(s, q, sms, ctas, smem)
                  : launch_t<Pol, true, false, true>(s, q, sms, ctas, smem);
    return site ? launch_t<Pol, true, true, false>(s, q, sms, ctas, smem)
                : launch_t<Pol, true, false, false>(s, q, sms, ctas, smem);
  }
  if (metric)
    return site ? launch_t<Pol, false, true, true>(s, q, sms, ctas, smem)
                : launch_t<Pol, false, false, true>(s, q, sms, ctas, smem);
  return site ? launch_t<Pol, false, true, false>(s, q, sms, ctas, smem)
              : launch_t<Pol, false, false, false>(s, q, sms, ctas, smem);
}

}  // namespace

cudaError_t run_block2d(cudaStream_t s, const Run2D& run, bool* done) {
  *done = false;
  const int pol = run.pol;
  Block2D q{};
  q.p = run.bank[0];
  q.counter = run.counter;
  q.d = run.dft;
  q.slots = run.slots;
  q.samples = run.samples;
  q.nsrc = run.nsrc;
  for (int n = 0; n < run.nsrc; ++n) {
    q.src[n] = run.src[n];
    q.timing[n] = run.timing[n];
  }
  q.nrec = run.nrec;
  for (int n = 0; n < run.nrec; ++n) q.rec[n] = run.rec[n];
  bool site = false;
  for (int c = 0; c < 3; ++c) site |= q.p.em.decay_full[c] || q.p.hm.decay_full[c] || q.p.hm.source_full[c];
  int device = 0, sms = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (err != cudaSuccess) return err;
  int T = std::min(run.steps_per_launch, run.nsteps);
  if (q.samples) T = std::min(T, run.batch / 2);
  T = std::max(1, std::min(T, kMaxT));
  Plan2D plan;
  while (!plan_tiles(q, pol, site, T, sms, &plan)) {
    if (T == 1) return cudaSuccess;  // not done: the caller steps one by one
    T = (T + 1) / 2;
  }
  // As many launches as put the result where nsteps single steps leave it.
  int launches = (run.nsteps + T - 1) / T;
  if ((launches & 1) != (run.nsteps & 1)) ++launches;
  int at = 0, prev = 0, planned = T;
  for (int n = 0; n < launches; ++n) {
    const int left = run.nsteps - at, count = (left + launches - n - 1) / (launches - n);
    if (count != planned) {
      if (!plan_tiles(q, pol, site, count, sms, &plan)) return cudaErrorInvalidConfiguration;
      planned = count;
    }
    Block2D b = q;
    b.p = run.bank[n & 1];
    b.g = plan.g;
    b.g.step_offset = at;
    b.g.slot0 = (n & 1) * (run.batch / 2);
    const int threads = launch_threads(b.g, sms);
    b.g.nflush = n > 0 && q.samples ? q.d.monitor_count * 3 * ((q.d.max_points + threads - 1) / threads) : 0;
    b.g.flush_first = at - prev;
    b.g.flush_count = prev;
    b.g.flush_slot0 = ((n + 1) & 1) * (run.batch / 2);
    const int ctas = b.g.nflush + b.g.gx * b.g.gy;
    err = pol == 0 ? launch_pol<0>(s, b, site, sms, ctas, plan.smem) : launch_pol<1>(s, b, site, sms, ctas, plan.smem);
    if (err != cudaSuccess) return err;
    at += count;
    prev = count;
  }
  if (q.samples) {
    const dim3 grid((q.d.max_points + 255) / 256, q.d.monitor_count * 3, 1);
    flush_raw_kernel<<<grid, 256, 0, s>>>(q.d, q.samples, q.counter, at - prev,
                                          ((launches - 1) & 1) * (run.batch / 2), prev, pol);
    err = cudaPeekAtLastError();
    if (err != cudaSuccess) return err;
  }
  finish_kernel<<<1, 1, 0, s>>>(run.counter, run.nsteps, q.nrec, q.rec[0], q.rec[1], q.rec[2],
                                q.rec[3]);
  err = cudaPeekAtLastError();
  *done = err == cudaSuccess;
  return err;
}

}  // namespace fdtd
