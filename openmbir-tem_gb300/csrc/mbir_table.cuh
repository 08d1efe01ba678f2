// mbir_table.cuh -- the table-driven ICD sweep and forward projection (FP32, three-bin
// footprints, one detector row per slice: every level whose voxels are detector pixels).
//
// The same updates in the same order as run_slice / group_step of mbir_sweep.cuh, operation for
// operation (the same bits), with everything that does not depend on the voxel taken out of the
// voxel step and everything that does not depend on the row's updates taken out of the row walk.
// One CTA owns one voxel slice, as there.
//
// What bounds it: a sweep is a chain of class steps with a CTA barrier after each, and every
// step is one warp's serial chain of instructions (the detector rows stay in shared memory), so
// both the step and the passage from one z-row to the next are written for few instructions and
// short dependence chains.
#pragma once
#include "mbir_sweep.cuh"

namespace mbir {
namespace sweep {

// ---- the voxel step ------------------------------------------------------------------------
// group_step issued ~1290 instructions per voxel pair (~1250 with the A-column table) at about
// one per 6 cycles, a dense 512 x 256 x 128 sweep of 61 views taking 19.4 ms; this one ~500 and
// 7.1 ms.  The A-column comes from the engine's table (16 bytes per view instead of ~60
// instructions), per-view constants and offsets stay in registers for the whole slice, the
// prior's constants are kernel arguments, footprint entries are read unconditionally and only
// their sums and stores are predicated, and the Bragg selector's rejected entries (rare) take a
// separate path.
template <int G, int VPL, bool BF>
struct TabCtx {
  const float4* acol;         // A-column table, at this lane's first view
  float* es;                  // error rows of the slice
  int eoff[VPL];              // this lane's views' rows in es (0 without a view)
  float gx[VPL];              // gain
  float gw[BF ? 1 : VPL];     // weight (HAADF)
  const float* bw;            // bright field: weights and selector rows of the slice
  uint8_t* bs;
  int woff[BF ? VPL : 1], soff[BF ? VPL : 1];
  float bt, bdt;
  unsigned long long* mag_fx;
  float hh;                   // t-response
  float* vol_y;               // the slice's plane
  int noff[2];                // this lane's neighbours: offset in the cache or in the volume
  int ndz[2], ndx[2];
  bool nok[2];                // the lane has that neighbour and its y lies in the volume
  bool nco[2];                // read past L1: another CTA of the launch writes that plane
  float nf[2];                // prior weight
};

template <int G, int VPL, bool STAGE, bool BF>
__device__ __forceinline__ void tab_ctx(TabCtx<G, VPL, BF>& c, const SweepArgs& A, int y,
                                        float* es, int rs, const float* bw, uint8_t* bs, int bs_rs,
                                        float hh, bool sched, bool coherent, int lane) {
  const DevGeom& g = A.g;
  const int gl = lane & (G - 1);
  const int plane = g.n_z * g.n_x;
  const float2* ggw = static_cast<const float2*>(A.tab.gw);
  c.acol = A.acol + gl;
  c.es = es;
  c.bw = bw;
  c.bs = bs;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int v = gl + G * i;
    const bool ok = v < g.n_theta;
    const float2 gw = ok ? ggw[v] : make_float2(0.f, 0.f);
    c.eoff[i] = ok ? v * rs : 0;
    c.gx[i] = gw.x;
    if constexpr (BF) {
      c.woff[i] = ok ? v * g.n_rp : 0;
      c.soff[i] = ok ? v * bs_rs : 0;
    } else {
      c.gw[i] = gw.y;
    }
  }
  c.bt = c.bdt = 0.f;
  c.mag_fx = nullptr;
  if constexpr (BF) {
    c.bt = static_cast<float>(A.bfa.bragg_t);
    c.bdt = static_cast<float>(A.bfa.bragg_dt);
    c.mag_fx = A.bfa.mag_fx;
  }
  c.hh = hh;
  c.vol_y = static_cast<float*>(A.x) + static_cast<size_t>(y) * plane;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int k = gl + G * i;
    const int dy = k / 9 - 1, dz = (k / 3) % 3 - 1, dx = k % 3 - 1;
    c.ndz[i] = dz;
    c.ndx[i] = dx;
    c.nok[i] = k < 27 && k != 13 && y + dy >= 0 && y + dy < g.n_y;
    c.nco[i] = coherent && dy != 0;
    c.noff[i] = sched ? dy * plane + dz * g.n_x + dx : ((dy + 1) * 3 + dz + 1) * g.n_x + dx;
    c.nf[i] = A.pf.f[k < 27 ? k : 0];
  }
}

// rho'(d)/d, the FP32 qggmrf_coef with the kernel's constants
__device__ __forceinline__ float qggmrf_coef_tab(const PriorF& q, float d0) {
  const float ad = fabsf(d0);
  const float t1 = __powf(ad, q.PQ) * q.inv_sig_pq;
  const float t3 = q.c + t1;
  float r = __fdividef(q.P * q.c + q.Q * t1, t3 * t3 * q.sp);
  if (q.P != 2.f) r *= __powf(ad, q.P - 2.f);
  return d0 == 0.f ? q.P / (q.sp * q.c) : r;
}

// The three weights at row[j..j+2], from 16-byte loads: rows in memory are whole 16 bytes, so the
// values lie in two windows of four, each read only when one of its values has a footprint value
// `a` (others are undefined).  A gather's lanes read neighbouring values of 32 different rows, and
// L1 takes about one row per clock, which bounds the classes of a bright-field call whose slices
// lie in HBM: 1.5 loads per view instead of 3 (and 1.25 instead of 3 for the selector), with the
// unchanged selector bytes not written, took six calls of the 1024 x 512 x 256 volume at 121 views
// from 158 to 115 ms.  Windows for the error as well: 117 ms; for weights of slices in shared
// memory 17.1 -> 19.8 ms, for HAADF errors 40.8 -> 50, for the coarse level's two rows 40 -> 60:
// there latency and instructions count, not the number of loads.
template <int NB>
__device__ __forceinline__ void gather_row(const float* row, int j, const float (&a)[NB],
                                           float (&out)[NB]) {
  static_assert(NB == 3, "two windows of four");
  const int k = j & ~3, off = j & 3;
  bool p0 = false, p1 = false;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    p0 |= a[b] > 0.f && off + b < 4;
    p1 |= a[b] > 0.f && off + b >= 4;
  }
  const float4* q = reinterpret_cast<const float4*>(row + k);
  float4 w0 = make_float4(0.f, 0.f, 0.f, 0.f), w1 = w0;
  if (p0) w0 = __ldg(q);
  if (p1) w1 = __ldg(q + 1);
  const float v[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
  float u[NB + 1];
#pragma unroll
  for (int b = 0; b <= NB; ++b) u[b] = (off & 2) ? v[b + 2] : v[b];
#pragma unroll
  for (int b = 0; b < NB; ++b) out[b] = (off & 1) ? u[b + 1] : u[b];
}
// The same for selector bytes (rows of whole 8 bytes, two windows of eight)
template <int NB>
__device__ __forceinline__ void gather_row(const uint8_t* row, int j, const float (&a)[NB],
                                           unsigned (&out)[NB]) {
  const int k = j & ~7, off = j & 7;
  bool p0 = false, p1 = false;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    p0 |= a[b] > 0.f && off + b < 8;
    p1 |= a[b] > 0.f && off + b >= 8;
  }
  const unsigned long long* q = reinterpret_cast<const unsigned long long*>(row + k);
  unsigned long long w0 = 0ull, w1 = 0ull;
  if (p0) w0 = q[0];
  if (p1) w1 = q[1];
  const unsigned long long w = off ? (w0 >> (8 * off)) | (w1 << (64 - 8 * off)) : w0;
#pragma unroll
  for (int b = 0; b < NB; ++b) out[b] = static_cast<unsigned>(w >> (8 * b)) & 0xffu;
}

// One updated voxel in the sweep's statistics, its line's magnitude for bright field
template <bool BF>
__device__ __forceinline__ void count_update(const SweepArgs& A, unsigned long long* mag_fx, int z,
                                             int x, float dlt, float V, GroupAcc& acc) {
  const DevGeom& g = A.g;
  const unsigned long long d = fix32<float>(dlt);
  if (x >= g.roi_x0 && x <= g.roi_x1 && z >= g.roi_z0 && z <= g.roi_z1) {
    acc.v[0] += d;
    acc.v[1] += fix32<float>(V);
  }
  acc.v[3] += 1;
  if constexpr (BF) {
    if (mag_fx != nullptr && dlt != 0.f) atomicAdd(mag_fx + z * g.n_x + x, d);
  }
}

// This lane's views of a voxel line's A-column (zeros for a group without a voxel)
template <int G, int VPL, bool BF>
__device__ __forceinline__ void table_load(const SweepArgs& A, const TabCtx<G, VPL, BF>& c,
                                           int line, bool active, int lane, float4 (&aq)[VPL]) {
  const int gl = lane & (G - 1), n_theta = A.g.n_theta;
  const float4* ac = c.acol + static_cast<size_t>(line) * n_theta;
#pragma unroll
  for (int i = 0; i < VPL; ++i)
    aq[i] = (active && gl + G * i < n_theta) ? __ldg(ac + G * i)
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
}

// One voxel (z, x) of the slice per group of G lanes; all 32 lanes of the warp call it together.
// SCHED: a scheduled call (neighbours from the volume); otherwise a row of the walk: neighbours
// from the row's cache, the new value into the cache, `touched` marked (row_end stores and
// counts).
template <int G, int VPL, bool STAGE, bool BF, bool SCHED>
__device__ __forceinline__ void table_step(const SweepArgs& A, const TabCtx<G, VPL, BF>& c, int z,
                                           int x, bool active, const float4 (&aq)[VPL],
                                           float* cache, uint8_t* touched, int lane, bool zs,
                                           GroupAcc& acc) {
  constexpr int NB = 3, NNB = (27 + G - 1) / G;
  const int gl = lane & (G - 1);
  const int n_x = A.g.n_x;
  const int line = z * n_x + x;
  // neighbours (UpdateVoxels.cpp:283-306); V last, so that a lane's loads are in flight together
  float nb[NNB];
  bool nv_ok[NNB];
  bool pos = false;
#pragma unroll
  for (int i = 0; i < NNB; ++i) {
    nv_ok[i] = c.nok[i] && static_cast<unsigned>(x + c.ndx[i]) < static_cast<unsigned>(n_x) &&
               static_cast<unsigned>(z + c.ndz[i]) < static_cast<unsigned>(A.g.n_z);
    nb[i] = 0.f;
    if (nv_ok[i]) {
      if constexpr (SCHED) {
        const float* src = c.vol_y + (line + c.noff[i]);
        nb[i] = c.nco[i] ? __ldcg(src) : *src;
      } else {
        nb[i] = cache[c.noff[i] + x];
      }
    }
    pos |= nb[i] > 0.f;
  }
  const float V = SCHED ? c.vol_y[line] : cache[4 * n_x + x];
  bool live = active;
  if (zs) {  // zero skipping at the visit; the ballot runs on all 32 lanes
    const bool any_pos = group_any<G>(pos, lane);
    if (V == 0.f && !any_pos) {
      if (active && gl == 0) acc.v[2] += 1;
      live = false;
    }
    if (!__any_sync(kFull, live)) return;
  }

  // footprint entries, all in flight together
  constexpr bool kWide = BF && !STAGE;  // weights and selector by windows (gather_row)
  float ev[VPL][NB];
  float wv[BF ? VPL : 1][NB];
  unsigned sv[BF ? VPL : 1][NB];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const int j = __float_as_int(aq[i].x);
    const float a[NB] = {aq[i].y, aq[i].z, aq[i].w};
    const float* er = c.es + (c.eoff[i] + j);
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      ev[i][b] = 0.f;
      if (STAGE || a[b] > 0.f) ev[i][b] = er[b];
    }
    if constexpr (kWide) {
      gather_row<NB>(c.bw + c.woff[i], j, a, wv[i]);
      gather_row<NB>(c.bs + c.soff[i], j, a, sv[i]);
    } else if constexpr (BF) {
      const float* wr = c.bw + (c.woff[i] + j);
      const uint8_t* sr = c.bs + (c.soff[i] + j);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        wv[i][b] = 0.f;
        if (a[b] > 0.f) wv[i][b] = __ldg(wr + b);
        sv[i][b] = sr[b];
      }
    }
  }

  // QGGMRF surrogate sums (QGGMRF_Functions.cpp:153-206): arithmetic under the loads above
  float s1 = 0.f, s2 = 0.f, lo = 0.f, hi = 0.f;
#pragma unroll
  for (int i = 0; i < NNB; ++i) {
    const float tc = c.nf[i] * qggmrf_coef_tab(A.pf, V - nb[i]);
    if (nv_ok[i]) {
      s1 += tc * nb[i];
      s2 += tc;
    }
    lo = nb[i] < lo ? nb[i] : lo;
    hi = nb[i] > hi ? nb[i] : hi;
  }

  // theta1 / theta2 (UpdateVoxels.cpp:343-369; BF: BFForwardModel.cpp:851-892)
  float t1 = 0.f, t2 = 0.f;
  // bit i * NB + b: selected before the update (kept where the registers are short), rejected
  unsigned on0 = 0, rejected = 0;
  auto was_on = [&](int i, int b) {
    return kWide ? on0 >> (i * NB + b) & 1u : sv[BF ? i : 0][b];
  };
  if constexpr (BF) {
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const unsigned bit = 1u << (i * NB + b);
        if (kWide && sv[i][b] != 0) on0 |= bit;
        if (f4_at(aq[i], b + 1) > 0.f && sv[i][b] == 0) rejected |= bit;
      }
  }
  if (!BF || !__any_sync(kFull, rejected != 0)) {
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const float a = f4_at(aq[i], b + 1);
        const float w = BF ? wv[BF ? i : 0][b] : c.gw[BF ? 0 : i];
        const float pe = c.gx[i] * a * c.hh;
        const float x2 = pe * pe * w, x1 = ev[i][b] * pe * w;
        if (a > 0.f) {
          t2 += x2;
          t1 += x1;
        }
      }
  } else if constexpr (BF) {
    // entries that the selector rejects count with weight delta T / (|e| sqrt(w)): a root and a
    // division, ~300 cycles of a chain that nothing overlaps.  The lanes take them together, each
    // for its own next rejected entry, as often as one lane has rejected entries instead of once
    // for each of its VPL * NB entries (20 calls at 75 views, T = 3: 14.5 -> 13.3 ms of sweep
    // kernels; at 61 views 17.1 -> 15.9)
    float qc[VPL * NB];
#pragma unroll
    for (int k = 0; k < VPL * NB; ++k) qc[k] = 0.f;
    while (rejected) {
      const unsigned bit = rejected & (0u - rejected);
      rejected ^= bit;
      float e = 0.f, w = 0.f;
#pragma unroll
      for (int k = 0; k < VPL * NB; ++k) {
        e = bit == (1u << k) ? ev[k / NB][k % NB] : e;
        w = bit == (1u << k) ? wv[k / NB][k % NB] : w;
      }
      const float q = c.bdt / (fabsf(e) * sqrtf(w));
#pragma unroll
      for (int k = 0; k < VPL * NB; ++k) qc[k] = bit == (1u << k) ? q : qc[k];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < VPL; ++i)
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const float a = f4_at(aq[i], b + 1);
        const float w = wv[i][b];
        const float pe = c.gx[i] * a * c.hh;
        if (a > 0.f) {
          if (was_on(i, b)) {
            t2 += pe * pe * w;
            t1 += ev[i][b] * pe * w;
          } else {
            t2 += qc[i * NB + b] * (pe * pe * w);
            t1 += qc[i * NB + b] * (ev[i][b] * pe * w);
          }
        }
      }
  }
  const float theta1 = -group_sum<G>(t1);
  const float theta2 = group_sum<G>(t2);
  lo = group_min<G>(lo);
  hi = group_max<G>(hi);
  s1 = group_sum<G>(s1);
  s2 = group_sum<G>(s2);
  // bracket, surrogate minimum, positivity (UpdateVoxels.cpp:47-63, 372-400)
  if (theta2 != 0.f) {
    const float cand = V - theta1 / theta2;
    lo = lo > cand ? cand : lo;
    hi = hi < cand ? cand : hi;
  }
  const float u = (s1 + theta2 * V - theta1) / (s2 + theta2);
  float nv = V + A.pf.alpha * (u - V);
  nv = (nv < lo) ? lo : ((nv > hi) ? hi : nv);
  if (nv < 0.f) nv = 0.f;
  const float dlt = nv - V;
  if (!live) return;
  // error-sinogram scatter (UpdateVoxels.cpp:423-449); BF re-evaluates the selector of every
  // footprint entry even when the voxel did not change (BFForwardModel.cpp:898-932)
  if (BF || dlt != 0.f) {
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      const int j = __float_as_int(aq[i].x);
      float* er = c.es + (c.eoff[i] + j);
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const float a = f4_at(aq[i], b + 1);
        const float ne = ev[i][b] - c.gx[i] * (a * c.hh * dlt);
        if (a > 0.f) {
          er[b] = ne;
          if constexpr (BF) {
            // the selector seldom changes: in HBM its byte is then not written (a fifth of the
            // call's time at 1024 bins and 121 views); in shared memory the test costs more than
            // the store (19.0 against 17.1 ms of sweep kernels per equivalent iteration)
            const unsigned on = bragg_selected<float>(ne, wv[i][b], c.bt);
            if (STAGE || on != was_on(i, b)) c.bs[c.soff[i] + j + b] = static_cast<uint8_t>(on);
          }
        }
      }
    }
  }
  if (gl == 0) {
    if constexpr (SCHED) {
      c.vol_y[line] = nv;
      count_update<BF>(A, c.mag_fx, z, x, dlt, V, acc);
    } else {
      cache[4 * n_x + x] = nv;
      touched[x] = 1;
    }
  }
}

// Projection of one voxel per group: its footprint added to the slice's rows
// (HAADF_ReconstructionEngine.cpp:636-691).
template <int G, int VPL, bool STAGE, bool BF>
__device__ __forceinline__ void table_project(const TabCtx<G, VPL, BF>& c, int x, bool active,
                                              const float4 (&aq)[VPL], const float* row) {
  const float V = active ? row[x] : 0.f;
  if (V == 0.f) return;
  // the entries of a voxel are distinct: all of them read before the first is written
  float ev[VPL][3];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    const float* er = c.es + (c.eoff[i] + __float_as_int(aq[i].x));
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (STAGE || f4_at(aq[i], b + 1) > 0.f) ev[i][b] = er[b];
  }
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    float* er = c.es + (c.eoff[i] + __float_as_int(aq[i].x));
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const float a = f4_at(aq[i], b + 1);
      if (a > 0.f) er[b] = ev[i][b] + c.gx[i] * (a * c.hh * V);
    }
  }
}

// ---- one slice -----------------------------------------------------------------------------
enum TableKind : int { kTable = 1, kTableProject = 2 };

// Shared memory of a table-driven slice.  nbuf: row caches (2 when they fit: the next row's
// neighbours arrive while the current row is updated).  Scheduled calls walk no rows (n_x = 0).
struct TableLayout {
  size_t bar, ctl, words, cls, list, flat, touched, vold, raw, cache, es, sel, stats, total;
  int nw, raw_stride, cache_rows;
};

constexpr int kStatRows = 32;  // warps of the largest CTA

__host__ __device__ inline TableLayout table_layout(int n_theta, int n_x, int n_rs, bool stage,
                                                    int n_sp, bool project, int nbuf) {
  TableLayout L;
  const size_t nx = static_cast<size_t>(n_x);
  size_t o = 0;
  L.bar = o;
  o += 16;
  L.ctl = o;  // [1] zero-skipped voxels
  o += 16;
  L.nw = (n_x + 31) / 32 + 2;  // one word of zeros before and after the row's
  L.words = o;                 // listed (ok), V != 0, column > 0, live, candidates
  o = align_up(o + sizeof(unsigned) * 5 * L.nw, 16);
  L.cls = o;  // per class (S <= max(n_x, 2)): its list's offset and length, then the classes that
              // it conflicts with
  o = align_up(o + 3 * sizeof(int) * (nx + 2), 16);
  L.list = o;  // class segments: S * ceil(n_x / S) <= 2 n_x + 2 slots
  o = align_up(o + sizeof(uint16_t) * (2 * nx + 2), 16);
  L.flat = o;  // the classes' candidates one class after another
  o = align_up(o + sizeof(uint16_t) * (nx + 2), 16);
  L.touched = o;
  o = align_up(o + nx, 16);
  L.vold = o;  // the row's values before its updates
  o = align_up(o + sizeof(float) * nx, 16);
  L.raw_stride = static_cast<int>(align_up(nx + 8, 16));
  L.raw = o;  // line flags of a row (whole words around it): non-empty column, in the call
  o = align_up(o + static_cast<size_t>(2 * nbuf) * L.raw_stride, 16);
  L.cache_rows = project ? 1 : 9;
  L.cache = o;
  o = align_up(o + sizeof(float) * nx * L.cache_rows * nbuf, 128);
  L.es = o;
  if (stage) o += sizeof(float) * static_cast<size_t>(n_theta) * n_rs;
  o = align_up(o, 16);
  L.sel = o;
  if (stage && n_sp > 0) o += static_cast<size_t>(n_theta) * n_sp;
  o = align_up(o, 16);
  // after the rows: table_step reads up to three entries before and after a view's row whether
  // or not the footprint has them, and those reads stay inside the layout
  L.stats = o;
  o += sizeof(unsigned long long) * kStatRows * kStatSlots;
  L.total = align_up(o, 16);
  return L;
}

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}
// any bit of [lo, hi] (word 0 of w holds bits 0..31)
__device__ __forceinline__ bool any_bits(const unsigned* w, int lo, int hi) {
  for (int k = lo >> 5; k <= (hi >> 5); ++k) {
    const int a = max(lo - (k << 5), 0), b = min(hi - (k << 5), 31);
    if (w[k] & ((0xffffffffu >> (31 - (b - a))) << a)) return true;
  }
  return false;
}
// bits [x, x + 31] (x >= -32; the words before and after the row are zero)
__device__ __forceinline__ unsigned bits_at(const unsigned* w, int x) {
  const int k = x >> 5;
  return __funnelshift_r(w[k], w[k + 1], x & 31);
}

// The arrival of row z's inputs in buffer `buf`: the nine neighbour rows (projections: the row
// itself), one warp per row, and, unless every line of the volume is updated, the line flags.
// Rows outside the volume are zeros.  Each thread waits for its own copies (cp_async_wait_all)
// before the barrier that publishes them.  (Bulk copies instead: their issue took the warp 1500
// cycles a row and the proxy fences before them every thread 900.)
__device__ __forceinline__ void row_fetch(const SweepArgs& A, const TableLayout& L,
                                          unsigned char* smem, int y, int z, int buf,
                                          const uint8_t* active_lines) {
  const DevGeom& g = A.g;
  const int n_x = g.n_x, tid = threadIdx.x, nthreads = blockDim.x;
  const int lane = tid & 31;
  float* cache = reinterpret_cast<float*>(smem + L.cache) + buf * L.cache_rows * n_x;
  const float* vol = static_cast<const float*>(A.x);
  for (int r = tid >> 5; r < L.cache_rows; r += nthreads >> 5) {
    const int yy = L.cache_rows == 9 ? y + r / 3 - 1 : y;
    const int zz = L.cache_rows == 9 ? z + r % 3 - 1 : z;
    float* dst = cache + r * n_x;
    if (yy < 0 || yy >= g.n_y || zz < 0 || zz >= g.n_z) {
      for (int x = lane; x < n_x; x += 32) dst[x] = 0.f;
      continue;
    }
    const float* src = vol + (static_cast<size_t>(yy) * g.n_z + zz) * n_x;
    if ((n_x & 3) == 0) {  // rows of whole 16 bytes
      for (int x = 4 * lane; x < n_x; x += 128) cp_async16(dst + x, src + x);
    } else {
      for (int x = lane; x < n_x; x += 32) cp_async4(dst + x, src + x);
    }
  }
  if (A.all_lines && active_lines == nullptr) return;
  // flags: whole words (the flag arrays are padded to a word)
  const int b0 = (z * n_x) & ~3, nwords = (z * n_x + n_x - b0 + 3) / 4;
  unsigned char* raw = smem + L.raw + 2 * buf * L.raw_stride;
  for (int k = tid; k < nwords; k += nthreads) {
    cp_async4(raw + 4 * k, A.tab.lineok + b0 + 4 * k);
    if (active_lines != nullptr) cp_async4(raw + L.raw_stride + 4 * k, active_lines + b0 + 4 * k);
  }
}

// The z-rows of one slice in the call's row order.  Each row: its candidates (voxels that are
// updated now, or that an update of their own row can make updatable) per conflict-free class,
// then the classes one after another.
//
// The passage from one row to the next is as much on the critical path as the class steps: with
// loads issued at the row's start, liveness by one thread per period and one warp forming the
// steps it took 6.6k cycles of a dense row's 51k (512 voxels, 61 views), and 6.6k-18k against 9
// steps of 2.2k on a 128 x 64 plane with 71 views.  So the next row's inputs arrive during this
// row's steps, and candidates, lists and conflicts come from ballots and bit windows of all warps.
template <int G, int VPL, bool STAGE, bool BF, int KIND>
__device__ __forceinline__ void walk_rows(const SweepArgs& A, const TableLayout& L, int nbuf,
                                          unsigned char* smem, const TabCtx<G, VPL, BF>& tc, int y,
                                          bool zs_on, GroupAcc& acc) {
  const DevGeom& g = A.g;
  const int n_x = g.n_x, n_z = g.n_z;
  const int tid = threadIdx.x, nthreads = blockDim.x, warp = tid >> 5, lane = tid & 31;
  const int n_warps = nthreads >> 5;
  constexpr int GPW = 32 / G;
  const int group = warp * GPW + lane / G, n_groups = n_warps * GPW;
  constexpr bool kProject = KIND == kTableProject;
  unsigned* ctl = reinterpret_cast<unsigned*>(smem + L.ctl);
  unsigned* w_ok = reinterpret_cast<unsigned*>(smem + L.words) + 1;  // words -1 and nw-2 are 0
  unsigned* w_nz = w_ok + L.nw;
  unsigned* w_pos = w_nz + L.nw;
  unsigned* w_live = w_pos + L.nw;
  unsigned* w_cand = w_live + L.nw;
  int2* steps = reinterpret_cast<int2*>(smem + L.cls);  // (offset, voxels) of each step
  unsigned* conf = reinterpret_cast<unsigned*>(steps + n_x + 2);
  uint16_t* list = reinterpret_cast<uint16_t*>(smem + L.list);
  uint16_t* flat = reinterpret_cast<uint16_t*>(smem + L.flat);
  uint8_t* touched = smem + L.touched;
  float* vold = reinterpret_cast<float*>(smem + L.vold);
  float* const cache0 = reinterpret_cast<float*>(smem + L.cache);
  const int mid = kProject ? 0 : 4 * n_x;
  const int S = A.stride, cap = (n_x + S - 1) / S;
  const unsigned inv_S = 0xffffffffu / static_cast<unsigned>(S) + 1u;  // x / S for x S < 2^32
  const int words = (n_x + 31) >> 5;
  const uint8_t* active_lines = BF ? A.bfa.active : nullptr;
  const bool flags = !A.all_lines || active_lines != nullptr;
  unsigned skipped = 0;
  for (int i = tid; i < 5 * L.nw; i += nthreads) w_ok[i - 1] = 0u;

  row_fetch(A, L, smem, y, A.row_order[0], 0, active_lines);
  int z_prev = -4;
  for (int rr = 0; rr <= n_z; ++rr) {
    const int buf = nbuf == 2 ? (rr & 1) : 0;
    const int z = rr < n_z ? A.row_order[rr] : -4;
    float* cache = cache0 + buf * L.cache_rows * n_x;
    float* cache_prev = cache0 + (nbuf == 2 ? (buf ^ 1) : 0) * L.cache_rows * n_x;
    cp_async_wait_all();
    __syncthreads();  // the row before is done, this row's inputs are there (with two buffers)
    // row end: the finished row's values to the volume (coalesced), its updates counted; a row
    // next to it has its old values in its cache: replaced
    if constexpr (!kProject) {
      if (rr > 0) {
        const bool patch = nbuf == 2 && rr < n_z && z_prev - z <= 1 && z - z_prev <= 1;
        float* out = tc.vol_y + static_cast<size_t>(z_prev) * n_x;
        for (int x = tid; x < n_x; x += nthreads) {
          const float v = cache_prev[mid + x];
          if (touched[x]) {
            out[x] = v;
            const float o = vold[x];
            count_update<BF>(A, tc.mag_fx, z_prev, x, v - o, o, acc);
          }
          if (patch) cache[(4 + z_prev - z) * n_x + x] = v;
        }
      }
    }
    if (rr == n_z) break;
    if (nbuf != 2 && rr > 0) {
      __syncthreads();
      row_fetch(A, L, smem, y, z, 0, active_lines);
      cp_async_wait_all();
      __syncthreads();
    }
    // the row's flags as bit words, one warp per word
    {
      const unsigned char* raw = smem + L.raw + 2 * buf * L.raw_stride + ((z * n_x) & 3);
      for (int x = tid; x < words * 32; x += nthreads) {
        bool ok = x < n_x, nz = false, pos = false;
        if (ok) {
          if (flags)
            ok = (A.all_lines || raw[x] != 0) &&
                 (active_lines == nullptr || raw[L.raw_stride + x] != 0);
          const float V = cache[mid + x];
          nz = V != 0.f;
          if constexpr (!kProject) {
            vold[x] = V;
            touched[x] = 0;
            if (zs_on) {
#pragma unroll
              for (int r = 0; r < 9; ++r) pos |= cache[r * n_x + x] > 0.f;
            }
          }
        }
        const unsigned bo = __ballot_sync(kFull, ok), bn = __ballot_sync(kFull, nz);
        const unsigned bp = __ballot_sync(kFull, pos);
        if (lane == 0) {
          w_ok[x >> 5] = bo;
          w_nz[x >> 5] = bn;
          w_pos[x >> 5] = bp;
        }
      }
    }
    __syncthreads();
    if (nbuf == 2 && rr + 1 < n_z)  // the buffer of the row before is free now
      row_fetch(A, L, smem, y, A.row_order[rr + 1], buf ^ 1, active_lines);
    // liveness at the start of the row: projection needs V != 0; an ICD voxel that would be
    // zero-skipped now (V == 0, no neighbour > 0) is not live.  A voxel skipped at the start of
    // its row can still be updated if a same-row neighbour processed before it became positive:
    // within a stride period [mS, mS+S) classes run left to right, so reachability is the
    // period's prefix-OR, and the period's last voxel also follows the next period's first one.
    // `dense`: so many candidates (N) that neighbouring classes practically always have some
    // within S of each other (N / S per class: 2 N^2 / (S n_x) close pairs expected), so that the
    // search for classes to merge is left out.  (Counted are the threads that saw one, N itself
    // while n_x is at most the CTA's threads.  In longer rows a thread may stand for several; the
    // line at sqrt(S n_x / 2), 78 of 4000 voxels at S = 3, is far below the threads, so that only
    // rows with that few candidates can fall on either side.  Results do not depend on it.)
    int any_cand = 0;
    bool dense = true;
    if (kProject || !zs_on) {
      for (int k = tid; k < words; k += nthreads) {
        const unsigned c = kProject ? (w_ok[k] & w_nz[k]) : w_ok[k];
        w_cand[k] = c;
        any_cand |= c != 0u;
      }
      any_cand = __syncthreads_or(any_cand);
      if constexpr (!kProject) dense = active_lines == nullptr;
    } else {
      for (int k = tid; k < words; k += nthreads) {
        const unsigned p = w_pos[k];
        const unsigned l = (p << 1) | (w_pos[k - 1] >> 31), r = (p >> 1) | (w_pos[k + 1] << 31);
        const unsigned v = w_ok[k] & (w_nz[k] | p | l | r);
        w_live[k] = v;
        any_cand |= v != 0u;
      }
      any_cand = __syncthreads_or(any_cand);  // (no live voxel: no candidate)
      if (any_cand) {
        int mine = 0;
        for (int x = tid; x < words * 32; x += nthreads) {
          const int k = x - static_cast<int>(__umulhi(static_cast<unsigned>(x), inv_S)) * S;
          bool c;
          if (S <= 31)
            c = (bits_at(w_live, x - 31) >> (31 - k)) != 0u;
          else
            c = any_bits(w_live, x - k, x);
          c |= k == S - 1 && ((bits_at(w_live, x) >> 1) & 1u);
          const unsigned b = __ballot_sync(kFull, c) & w_ok[x >> 5];
          if (lane == 0) {
            w_cand[x >> 5] = b;
            skipped += __popc(w_ok[x >> 5] & ~b);
          }
          mine |= (b >> lane) & 1u;
        }
        const int count = __syncthreads_count(mine);
        dense = count * count >= S * n_x / 2;
      } else {
        for (int k = tid; k < words; k += nthreads) skipped += __popc(w_ok[k]);
      }
    }
    if (!any_cand) {
      z_prev = z;
      continue;
    }
    const bool merge = !dense && S <= 31;  // (strides that fit a mask word)
    // Warp w lists the candidates of classes w, w + warps, ... in ascending x, with the earlier
    // classes that have a candidate within S of one of theirs: in the window of S - 1 positions
    // before and after position x of class k, index i = 1..S-1 (from x - S, from x) is class
    // (k + i) mod S.
    for (int k = warp; k < S; k += n_warps) {
      int base = 0;
      unsigned cm = 0u;
      for (int m0 = 0; k + S * m0 < n_x; m0 += 32) {
        const int x = k + S * (m0 + lane);
        const bool cand = x < n_x && ((w_cand[x >> 5] >> (x & 31)) & 1u);
        const unsigned b = __ballot_sync(kFull, cand);
        if (cand) {
          list[k * cap + base + __popc(b & ((1u << lane) - 1u))] = static_cast<uint16_t>(x);
          if (merge) {
            const unsigned u = (bits_at(w_cand, x - S) | bits_at(w_cand, x)) &
                               ((1u << S) - 2u);
            cm |= u >> (S - k);  // the classes before k
          }
        }
        base += __popc(b);
      }
      if (merge) cm = __reduce_or_sync(kFull, cm);
      if (lane == 0) {
        steps[k] = make_int2(k * cap, base);
        conf[k] = cm;
      }
    }
    __syncthreads();
    // Steps: a class is a step (an empty one is passed over); in sparse rows consecutive classes
    // are merged while none of the next class's candidates lies within S of a candidate already
    // in the step: voxels of one step are then pairwise independent (no shared detector bin, no
    // prior neighbours, no zero-skipping influence), and independent updates commute, so a step
    // gives exactly the result of running its classes in order.  Every warp forms the steps:
    // lane k holds class k, `starts` has a bit for each class that opens a step, `pre` the
    // candidates of the classes before the lane's.
    int n_steps = S;
    const uint16_t* items = list;
    if (merge) {
      const int n_k = lane < S ? steps[lane].y : 0;
      const unsigned c_k = lane < S ? conf[lane] : 0u;
      unsigned left = __ballot_sync(kFull, n_k > 0);
      const unsigned used = left;
      unsigned starts = 0u, cur = 0u;
      while (left) {
        const int k = __ffs(left) - 1;
        const unsigned c = __shfl_sync(kFull, c_k, k);
        left &= left - 1u;
        if (cur == 0u || (c & cur)) {
          starts |= 1u << k;
          cur = 0u;
        }
        cur |= 1u << k;
      }
      if (starts != used) {
        int pre = n_k;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(kFull, pre, o);
          if (lane >= o) pre += t;
        }
        pre -= n_k;
        for (int k = warp; k < S; k += n_warps) {
          const int n = __shfl_sync(kFull, n_k, k), at = __shfl_sync(kFull, pre, k);
          for (int j = lane; j < n; j += 32) flat[at + j] = list[k * cap + j];
        }
        const unsigned later = starts & ~((2u << lane) - 1u);
        const int end = __shfl_sync(kFull, pre, later ? __ffs(later) - 1 : 31);
        __syncthreads();  // every warp has read the classes
        if (warp == 0 && ((starts >> lane) & 1u))
          steps[__popc(starts & ((1u << lane) - 1u))] = make_int2(pre, end - pre);
        __syncthreads();
        n_steps = __popc(starts);
        items = flat;
      }
    }
    // The group's voxels of consecutive rounds, the next one's A-column in flight while this one
    // is updated (it depends on no update): HAADF at 141 views with its slices in HBM 67.7 ->
    // 39.4 ms for three sweeps, staged slices 7.5 -> 7.1 ms a dense sweep.  Bright field has no
    // registers for it.
    constexpr bool kAhead = !BF;
    const int line0 = z * n_x;
    int st = 0, b0 = group;
    int2 cur = steps[0];
    while (cur.y == 0) cur = steps[++st];  // (some class has a candidate)
    bool act = b0 < cur.y;
    int x = act ? items[cur.x + b0] : 0;
    float4 aq[VPL];
    table_load<G, VPL, BF>(A, tc, line0 + x, act, lane, aq);
    for (;;) {
      int st2 = st;
      int2 nxt = cur;
      b0 += n_groups;
      if (b0 - group >= cur.y) {
        b0 = group;
        do nxt = ++st2 < n_steps ? steps[st2] : make_int2(0, -1);
        while (nxt.y == 0);
      }
      const bool act2 = b0 < nxt.y;
      const int x2 = act2 ? items[nxt.x + b0] : 0;
      float4 aq2[VPL];
      if constexpr (kAhead) table_load<G, VPL, BF>(A, tc, line0 + x2, act2, lane, aq2);
      if constexpr (kProject)
        table_project<G, VPL, STAGE, BF>(tc, x, act, aq, cache + mid);
      else
        table_step<G, VPL, STAGE, BF, false>(A, tc, z, x, act, aq, cache, touched, lane, zs_on,
                                             acc);
      if (nxt.y < 0) break;  // (the barrier after the last step: at the next row)
      if constexpr (!kAhead) table_load<G, VPL, BF>(A, tc, line0 + x2, act2, lane, aq2);
      if (st2 != st) __syncthreads();
      st = st2;
      cur = nxt;
      act = act2;
      x = x2;
#pragma unroll
      for (int i = 0; i < VPL; ++i) aq[i] = aq2[i];
    }
    z_prev = z;
  }
  if (skipped) atomicAdd(ctl + 1, skipped);
}

// A scheduled bright-field call: its lines class by class, one CTA barrier per class.  Neighbours
// come from the volume (the slice's own plane is written only by this CTA, the planes y+-1 belong
// to the other colour and do not change during the launch), the zero-skipping test runs at the
// visit.
template <int G, int VPL, bool STAGE, bool BF>
__device__ __forceinline__ void run_schedule(const SweepArgs& A, const TableLayout& L,
                                             unsigned char* smem, const TabCtx<G, VPL, BF>& tc,
                                             bool zs_on, GroupAcc& acc) {
  const int n_x = A.g.n_x;
  const int tid = threadIdx.x, nthreads = blockDim.x, warp = tid >> 5, lane = tid & 31;
  constexpr int GPW = 32 / G;
  const int group = warp * GPW + lane / G, n_groups = (nthreads >> 5) * GPW;
  const int n_levels = A.sched_count != nullptr ? __ldg(A.sched_count + 1) : A.n_levels;
  const int n_sl = __ldg(A.sched_lofs + n_levels);
  // the schedule (offsets, lines as z << 16 | x) in shared memory when it fits behind the layout
  int* s_lofs = nullptr;
  int* s_zx = nullptr;
  if (L.total + (static_cast<size_t>(n_levels) + 1 + n_sl) * sizeof(int) <= dynamic_smem_bytes()) {
    s_lofs = reinterpret_cast<int*>(smem + L.total);
    s_zx = s_lofs + n_levels + 1;
    for (int i = tid; i <= n_levels; i += nthreads) s_lofs[i] = __ldg(A.sched_lofs + i);
    for (int i = tid; i < n_sl; i += nthreads) {
      const int l = __ldg(A.sched_lines + i);
      const int z = l / n_x;
      s_zx[i] = (z << 16) | (l - z * n_x);
    }
    __syncthreads();
  }
  auto lofs_at = [&](int i) { return s_lofs ? s_lofs[i] : __ldg(A.sched_lofs + i); };
  auto zx_at = [&](int i) {  // line i of the schedule as z << 16 | x
    if (s_zx) return s_zx[i];
    const int l = __ldg(A.sched_lines + i);
    const int z = l / n_x;
    return (z << 16) | (l - z * n_x);
  };
  // (the next voxel's A-column is not loaded ahead here, as the row walk does: beside the weights
  // and selector bytes it does not fit the registers; 20.0 ms of sweep kernels per equivalent
  // iteration against 18.4 without)
  int b = lofs_at(0);
  for (int lv = 0; lv < n_levels; ++lv) {
    const int e = lofs_at(lv + 1);
    for (int b0 = b; b0 < e; b0 += n_groups) {
      const bool act = b0 + group < e;
      const int zx = act ? zx_at(b0 + group) : 0;
      const int z = zx >> 16, x = zx & 0xffff;
      float4 aq[VPL];
      table_load<G, VPL, BF>(A, tc, z * n_x + x, act, lane, aq);
      table_step<G, VPL, STAGE, BF, true>(A, tc, z, x, act, aq, nullptr, nullptr, lane, zs_on, acc);
    }
    b = e;
    __syncthreads();
  }
}

// One voxel slice y of one reconstruction, processed by the whole CTA; `phase`, `coherent`,
// `stat_out` and the result as for run_slice.
template <int G, int VPL, bool STAGE, bool BF, int KIND>
__device__ __forceinline__ bool run_table_slice(const SweepArgs& A, int y, unsigned char* smem,
                                                uint32_t& phase, bool coherent,
                                                double* stat_out) {
  const DevGeom& g = A.g;
  const int tid = threadIdx.x, nthreads = blockDim.x, warp = tid >> 5, lane = tid & 31;
  constexpr bool kProject = KIND == kTableProject;
  const int n_sp = BF ? A.bfa.n_sp : 0;
  const int tfirst = A.tab.t_first[y];
  const bool sched = BF && !kProject && A.sched_lines != nullptr;
  int nbuf = 1;
  TableLayout L = table_layout(g.n_theta, sched ? 0 : g.n_x, A.n_rs, STAGE, n_sp, kProject, 2);
  if (sched || L.total <= dynamic_smem_bytes())
    nbuf = 2;
  else
    L = table_layout(g.n_theta, g.n_x, A.n_rs, STAGE, n_sp, kProject, 1);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L.bar);
  unsigned* ctl = reinterpret_cast<unsigned*>(smem + L.ctl);
  const size_t sino_plane = static_cast<size_t>(g.n_theta) * g.n_rp;
  const size_t sel_plane = static_cast<size_t>(g.n_theta) * n_sp;
  float* const ge = static_cast<float*>(A.e) + static_cast<size_t>(tfirst) * sino_plane;
  uint8_t* const gs = BF ? A.bfa.sel + static_cast<size_t>(tfirst) * sel_plane : nullptr;
  const uint32_t row_bytes = static_cast<uint32_t>(g.n_rp * sizeof(float));
  float* es = ge;
  uint8_t* ss = gs;
  int rs = g.n_rp;
  if (tid < 4) ctl[tid] = 0u;
  if constexpr (STAGE) {
    es = reinterpret_cast<float*>(smem + L.es);
    rs = A.n_rs;
    if (BF) ss = smem + L.sel;
    if constexpr (kProject) {
      for (int i = tid; i < g.n_theta * rs; i += nthreads) es[i] = 0.f;
    } else {
      if (tid == 0)
        mbar_expect_tx(bar, static_cast<uint32_t>(g.n_theta) * (row_bytes + (BF ? n_sp : 0)));
      __syncthreads();
      for (int v = tid; v < g.n_theta; v += nthreads) {
        bulk_g2s(es + v * rs, ge + static_cast<size_t>(v) * g.n_rp, row_bytes, bar);
        if (BF)
          bulk_g2s(ss + v * n_sp, gs + static_cast<size_t>(v) * n_sp, static_cast<uint32_t>(n_sp),
                   bar);
      }
      const bool ok = mbar_wait(bar, phase);
      phase ^= 1u;
      if (!__syncthreads_and(ok)) {
        if (tid == 0) atomicOr(A.err, 1);
        mbar_wait(bar, phase ^ 1u);  // give copies still in flight a second bounded chance
        return false;
      }
    }
  }
  __syncthreads();
  const bool zs_on = !kProject && A.zero_skipping && A.iter_nonzero;
  TabCtx<G, VPL, BF> tc;
  tab_ctx<G, VPL, STAGE, BF>(
      tc, A, y, es, rs,
      BF ? static_cast<const float*>(A.bfa.w) + static_cast<size_t>(tfirst) * sino_plane : nullptr,
      ss, n_sp, static_cast<const float*>(A.tab.hval)[y * kMaxTRows], sched, coherent, lane);
  GroupAcc acc;
#pragma unroll
  for (int s = 0; s < kStatSlots; ++s) acc.v[s] = 0ull;
  if constexpr (BF && !kProject) {
    if (sched)
      run_schedule<G, VPL, STAGE, BF>(A, L, smem, tc, zs_on, acc);
    else
      walk_rows<G, VPL, STAGE, BF, KIND>(A, L, nbuf, smem, tc, y, zs_on, acc);
  } else {
    walk_rows<G, VPL, STAGE, BF, KIND>(A, L, nbuf, smem, tc, y, zs_on, acc);
  }

  if constexpr (STAGE) {
    fence_proxy_async_smem();
    __syncthreads();
    for (int v = tid; v < g.n_theta; v += nthreads) {
      bulk_s2g(ge + static_cast<size_t>(v) * g.n_rp, es + v * rs, row_bytes);
      if (BF && !kProject)
        bulk_s2g(gs + static_cast<size_t>(v) * n_sp, ss + v * n_sp, static_cast<uint32_t>(n_sp));
    }
    bulk_commit();
    bulk_wait_all();
  }
  if (stat_out != nullptr) {
    // integer sums, so the order does not matter
    unsigned long long* sstat = reinterpret_cast<unsigned long long*>(smem + L.stats);
#pragma unroll
    for (int s = 0; s < kStatSlots; ++s) {
      const unsigned long long t = group_sum<32>(acc.v[s]);
      if (lane == 0) sstat[warp * kStatSlots + s] = t;
    }
    __syncthreads();
    if (tid < kStatSlots) {
      unsigned long long t = 0;
      for (int w = 0; w < nthreads / 32; ++w) t += sstat[w * kStatSlots + tid];
      if (tid == 2) t += ctl[1];
      stat_out[tid] = tid < 2 ? static_cast<double>(t) / kFixScale : static_cast<double>(t);
    }
  }
  __syncthreads();
  return true;
}

// Threads of a CTA.  The step needs ~120 registers: with 640 or 768 threads (96 or 80 registers)
// it spills, 8.7 and 11.3 ms a dense sweep against 7.1.  A projection has fewer live values: 768
// threads take 4.9 ms for a dense 512 x 256 x 128 volume, 512 take 5.3.
constexpr int table_threads(int kind) { return kind == kTableProject ? 768 : kWarps * 32; }

// One launch = the slices of one y-colour of one reconstruction, one CTA per slice.
template <int G, int VPL, bool STAGE, bool BF, int KIND>
__global__ void __launch_bounds__(table_threads(KIND), 1)
    table_kernel(const __grid_constant__ SweepArgs A) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int y = (A.y_end > 0 ? A.y_first : A.colour) + 2 * static_cast<int>(blockIdx.x);
  if (y >= (A.y_end > 0 ? A.y_end : A.g.n_y)) return;
  init_slice_barrier(smem);
  uint32_t phase = 0;
  run_table_slice<G, VPL, STAGE, BF, KIND>(
      A, y, smem, phase, false,
      A.stats != nullptr ? A.stats + static_cast<size_t>(blockIdx.x) * kStatSlots : nullptr);
}

template <int G, int VPL, bool STAGE, bool BF, int KIND>
int launch_table_t(const SweepArgs& a, size_t smem, cudaStream_t s) {
  return launch_slices<table_kernel<G, VPL, STAGE, BF, KIND>>(a, smem, table_threads(KIND), s);
}

template <bool STAGE, bool BF, int KIND>
int launch_table_kind(const SweepArgs& a, int shape, size_t smem, cudaStream_t s) {
  if (shape == 1) return launch_table_t<16, 4, STAGE, BF, KIND>(a, smem, s);
  if (shape == 2) return launch_table_t<32, 2, STAGE, BF, KIND>(a, smem, s);
  if (shape == 3) return launch_table_t<32, 3, STAGE, BF, KIND>(a, smem, s);
  if (shape == 4) return launch_table_t<32, 5, STAGE, BF, KIND>(a, smem, s);
  if constexpr (!STAGE) return launch_table_t<32, 8, STAGE, BF, KIND>(a, smem, s);
  return -7;
}

// shape (1..5) when it covers the views, else the default for the view count
template <bool BF>
int launch_table_pick(const SweepArgs& a, size_t smem, cudaStream_t s) {
  const int shape = resolved_shape(a.shape, a.g.n_theta);
  const bool project = a.mode == kModeProject;
  if constexpr (!BF) {
    if (project)
      return a.smem_rows ? launch_table_kind<true, false, kTableProject>(a, shape, smem, s)
                         : launch_table_kind<false, false, kTableProject>(a, shape, smem, s);
  } else {
    if (project) return -7;
  }
  return a.smem_rows ? launch_table_kind<true, BF, kTable>(a, shape, smem, s)
                     : launch_table_kind<false, BF, kTable>(a, shape, smem, s);
}

// The persistent batched sweep (batch_sweep_kernel) of table-driven series, staged or not in
// separate launches.  It still spills where the same step launched alone does not (0 to 52 bytes of
// stores a thread up to 160 views): the arguments come from a shared copy instead of the constant
// bank, and bright field holds the row walk and the scheduled call in one kernel.  Bytes of spill
// stores staged / in HBM: bright field 16 x 4 356 / 388, 32 x 2 48 / 28, 32 x 3 164 / 148, 32 x 5
// 480 / 508; HAADF 108 / 96, 8 / 0, 16 / 4, 120 / 100.
template <int G, int VPL, bool STAGE, bool BF>
__global__ void __launch_bounds__(kWarps * 32, 1) batch_table_kernel(BatchArgs B) {
  batch_items(B, [](const SweepArgs& sA, int y, unsigned char* smem, uint32_t& phase,
                    double* stat_out) {
    run_table_slice<G, VPL, STAGE, BF, kTable>(sA, y, smem, phase, true, stat_out);
  });
}

template <bool STAGE, bool BF>
int launch_batch_table(const BatchArgs& b, int shape, int threads, size_t smem, int grid,
                       cudaStream_t s) {
  if (shape == 1)
    return launch_batch_kernel<batch_table_kernel<16, 4, STAGE, BF>>(b, smem, grid, threads, s);
  if (shape == 2)
    return launch_batch_kernel<batch_table_kernel<32, 2, STAGE, BF>>(b, smem, grid, threads, s);
  if (shape == 3)
    return launch_batch_kernel<batch_table_kernel<32, 3, STAGE, BF>>(b, smem, grid, threads, s);
  return launch_batch_kernel<batch_table_kernel<32, 5, STAGE, BF>>(b, smem, grid, threads, s);
}

}  // namespace sweep
}  // namespace mbir
