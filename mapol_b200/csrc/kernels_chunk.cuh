// Kernels that keep a chunk of G lanes (cases) on one block for a whole solve (sm_100a).
//
// Cases are independent, so a block that owns G lanes of a group can walk every level of
// the elimination tree by itself: block barriers separate the levels, no block waits for
// another, and the launch per level (and class of front size) of the level-synchronous
// kernels, with its latency and its tail, disappears.
//
// What bounds such a walk is latency: a level is a handful of tiny fronts, and each would
// be a chain of round trips to L2 (task, indices, panel).  So x and the carried entries stay
// in shared memory (where they fit), and everything a level reads that no level writes (its
// panels and index lists, stored in the order of the walk) streams through a ring buffer in
// shared memory with cp.async, two steps ahead.  A step then costs a barrier and its
// arithmetic.  Small supernodes (most of them) take 1 to 8 threads per lane without barriers,
// and the few larger fronts of a step run beside them on teams of 32 to 512 threads.
#pragma once

#include "internal.h"
#include "kernels.cuh"

namespace mpfk {

using mpf::kChunkThreads;
using mpf::kRingSlots;
using mpf::kSoloPivots;
using mpf::SweepStep;

struct DevSweep {
  const int4* step;      // per step: e0, ne, i0, ni
  const int* step_ptr;   // steps of each island
  const int* down_ptr;   // of them, the first root-to-leaves step
  const int* idx;
};

// rows of the mismatch by island
struct ChunkRows {
  const int* rows;
  const int* ptr;  // [islands + 1]
};

// A team's barrier: a warp, or a named barrier (1 .. 15) of `team` threads; the whole
// block uses barrier 0
__device__ __forceinline__ void chunk_sync(int team, int bar) {
  if (team == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(team) : "memory");
}

// x and the carried entries of a chunk: entry i of this thread's lane at x[i * S], c[i * S]
// (shared memory: S = G; the LU system's arrays: S = 32)
template <typename T>
struct ChunkVec {
  T* x;
  T* c;
};

// One substitution step of a supernode.  Leaves to root (UP): L y = b, or with TR U^T z = b,
// the rows below the pivots carried to the parent; root to leaves: U x = y, or with TR
// L^T l = z, the ancestors' values known.
//
// solo: by `split` threads per lane (thread r of them, G apart in the warp), each with the
// pivots' values in registers and every split-th of the other rows.  All threads of the warp
// call it together (on: this one has a task).  pan: the task's panel at this lane, entries G
// apart.  The loops are kept rolled: a block runs each path once per step, so a kernel larger
// than the instruction cache is bound by fetching it (334 KB unrolled: 150k cycles per half
// step of a 300-bus fast-decoupled solve).
template <typename T, int G, int S, bool UP, bool TR>
__device__ __forceinline__ void solo_subst(bool on, int4 h, const int* ib, int r, int split, const T* pan,
                                           const ChunkVec<T>& v) {
  constexpr int W = kSoloPivots;
  const int w = on ? h.y & 0xffff : 0, f = on ? h.y >> 16 : 0;
  const int* xi = ib + h.z + (UP ? 2 : 0);
  // entry (a, b) of the pivot block; row / column i beside it: entries sa apart from pivot to
  // pivot, at side0 + i si
  const int sa = UP == TR ? f * G : G, si = UP == TR ? G : w * G;
  const T* side0 = UP == TR ? pan : pan + (w * f - w * w) * G;
  T y[W];
  if (UP) {
    const int2* pr = reinterpret_cast<const int2*>(xi + ((w + 1) & ~1));
    const int layers = on ? xi[-2] : 0;
    auto carried = [&](int i, T s) {
#pragma unroll 1
      for (int k = 0; k < layers; ++k) {
        const int2 q = pr[k * f + i];
        if (q.x >= 0) s += v.c[q.x * S];
        if (q.y >= 0) s += v.c[q.y * S];
      }
      return s;
    };
#pragma unroll
    for (int a = 0; a < W; ++a) {
      y[a] = (T)0;
      if (a < w) {
        y[a] = carried(a, v.x[xi[a] * S]);
#pragma unroll
        for (int b = 0; b < a; ++b) y[a] -= pan[(TR ? b * f + a : a * f + b) * G] * y[b];
        if (TR) y[a] = y[a] / pan[(a * f + a) * G];
      }
    }
    if (on && h.w >= 0) {
#pragma unroll 1
      for (int i = w + r; i < f; i += split) {
        T s = carried(i, (T)0);
        const T* e = side0 + i * si;
#pragma unroll
        for (int a = 0; a < W; ++a)
          if (a < w) s -= e[a * sa] * y[a];
        v.c[(h.w + i - w) * S] = s;
      }
    }
    __syncwarp();  // the other threads of the task have read x
  } else {
    T acc[W];
#pragma unroll
    for (int a = 0; a < W; ++a) acc[a] = (T)0;
#pragma unroll 1
    for (int i = w + r; i < f; i += split) {
      const T xv = v.x[xi[i] * S];
      const T* e = side0 + i * si;
#pragma unroll
      for (int a = 0; a < W; ++a)
        if (a < w) acc[a] += e[a * sa] * xv;
    }
#pragma unroll 1
    for (int o = G; o < split * G; o <<= 1) {
#pragma unroll
      for (int a = 0; a < W; ++a) acc[a] += __shfl_xor_sync(0xffffffffu, acc[a], o);
    }
#pragma unroll
    for (int a = W - 1; a >= 0; --a) {
      y[a] = (T)0;
      if (a < w) {
        y[a] = v.x[xi[a] * S] - acc[a];
#pragma unroll
        for (int b = a + 1; b < W; ++b)
          if (b < w) y[a] -= pan[(TR ? b * f + a : a * f + b) * G] * y[b];
        if (!TR) y[a] = y[a] / pan[(a * f + a) * G];
      }
    }
    __syncwarp();
  }
  if (r == 0) {
#pragma unroll
    for (int a = 0; a < W; ++a)
      if (a < w) v.x[xi[a] * S] = y[a];
  }
}

// team: slot = thread / G, lane = thread % G; xs: the front's vector, [f][G]; us: the panel,
// entries es apart.  The pivots
// run one team barrier each; the rows that no later pivot needs take their whole sum
// without barriers.
template <typename T, int G, int S, bool UP, bool TR>
__device__ __forceinline__ void team_subst(int4 h, const int* xi, int team, int tid, int bar, T* xs, const T* us, int es,
                                           const ChunkVec<T>& v) {
  const int w = h.y & 0xffff, f = h.y >> 16, m = f - w;
  const int SL = team / G, slot = tid / G;  // shifts: G is a power of two
  if (UP) xi += 2;
  if (UP) {
    const int layers = xi[-2];
    const int2* pr = reinterpret_cast<const int2*>(xi + ((w + 1) & ~1));
#pragma unroll 1
    for (int i = slot; i < f; i += SL) {
      T b = i < w ? v.x[xi[i] * S] : (T)0;
#pragma unroll 1
      for (int k = 0; k < layers; ++k) {
        const int2 q = pr[k * f + i];
        if (q.x >= 0) b += v.c[q.x * S];
        if (q.y >= 0) b += v.c[q.y * S];
      }
      xs[i * G] = b;
    }
  } else {
#pragma unroll 1
    for (int q = slot; q < f; q += SL) xs[q * G] = v.x[xi[q] * S];
  }
  chunk_sync(team, bar);
  const T* ul = us + w * f * es;  // L panel below the diagonal block
  if (UP && !TR) {
#pragma unroll 1
    for (int p = 0; p + 1 < w; ++p) {
      const T yp = xs[p * G];
#pragma unroll 1
      for (int i = p + 1 + slot; i < w; i += SL) xs[i * G] -= us[(i * f + p) * es] * yp;
      chunk_sync(team, bar);
    }
#pragma unroll 1
    for (int i = slot; i < m; i += SL) {
      T b = xs[(w + i) * G];
#pragma unroll 2
      for (int p = 0; p < w; ++p) b -= ul[(i * w + p) * es] * xs[p * G];
      xs[(w + i) * G] = b;
    }
  } else if (UP) {
#pragma unroll 1
    for (int p = 0; p < w; ++p) {
      const T zp = xs[p * G] / us[(p * f + p) * es];
#pragma unroll 1
      for (int i = p + 1 + slot; i < w; i += SL) xs[i * G] -= us[(p * f + i) * es] * zp;
      chunk_sync(team, bar);
      if (slot == 0) xs[p * G] = zp;
    }
    chunk_sync(team, bar);
#pragma unroll 1
    for (int i = w + slot; i < f; i += SL) {
      T b = xs[i * G];
#pragma unroll 2
      for (int p = 0; p < w; ++p) b -= us[(p * f + i) * es] * xs[p * G];
      xs[i * G] = b;
    }
  } else if (!TR) {
#pragma unroll 1
    for (int r = slot; r < w; r += SL) {
      T a = xs[r * G], a2 = (T)0;
      const T* ur = us + r * f * es;
      int q = w;
#pragma unroll 1
      for (; q + 1 < f; q += 2) {
        a -= ur[q * es] * xs[q * G];
        a2 -= ur[(q + 1) * es] * xs[(q + 1) * G];
      }
      if (q < f) a -= ur[q * es] * xs[q * G];
      xs[r * G] = a + a2;
    }
    chunk_sync(team, bar);
#pragma unroll 1
    for (int p = w - 1; p >= 0; --p) {
      const T xp = xs[p * G] / us[(p * f + p) * es];
#pragma unroll 1
      for (int r = slot; r < p; r += SL) xs[r * G] -= us[(r * f + p) * es] * xp;
      chunk_sync(team, bar);
      if (slot == 0) xs[p * G] = xp;
    }
    chunk_sync(team, bar);
  } else {
#pragma unroll 1
    for (int p = slot; p < w; p += SL) {
      T a = xs[p * G], a2 = (T)0;
      int i = 0;
#pragma unroll 1
      for (; i + 1 < m; i += 2) {
        a -= ul[(i * w + p) * es] * xs[(w + i) * G];
        a2 -= ul[((i + 1) * w + p) * es] * xs[(w + i + 1) * G];
      }
      if (i < m) a -= ul[(i * w + p) * es] * xs[(w + i) * G];
      xs[p * G] = a + a2;
    }
    chunk_sync(team, bar);
#pragma unroll 1
    for (int p = w - 1; p > 0; --p) {
      const T xp = xs[p * G];
#pragma unroll 1
      for (int r = slot; r < p; r += SL) xs[r * G] -= us[(p * f + r) * es] * xp;
      chunk_sync(team, bar);
    }
  }
#pragma unroll 1
  for (int p = slot; p < w; p += SL) v.x[xi[p] * S] = xs[p * G];
  if (UP && h.w >= 0)
#pragma unroll 1
    for (int a = slot; a < m; a += SL) v.c[(h.w + a) * S] = xs[(w + a) * G];
  chunk_sync(team, bar);
}

// The block's ring buffer: kRingSlots slots of `slot` bytes
struct Ring {
  unsigned char* base;
  int slot;
};

// Starts the copies of step rec (e0, ne, i0, ni) into slot k and closes their group
template <typename T, int G>
__device__ __forceinline__ void ring_issue(const Ring& R, int k, int4 rec, const int* idx, const T* pan0) {
  constexpr int V = (int)(16 / sizeof(T)) < G ? (int)(16 / sizeof(T)) : G;
  constexpr int NV = G / V;
  unsigned char* at = R.base + (size_t)k * R.slot;
  const T* src = pan0 + (size_t)rec.x * 32;
#pragma unroll 1
  for (int i = threadIdx.x; i < rec.y * NV; i += kChunkThreads)
    cp_async<T, V>(reinterpret_cast<T*>(at) + (size_t)i * V, src + (size_t)(i / NV) * 32 + (i % NV) * V);
  int* di = reinterpret_cast<int*>(at + ((size_t)rec.y * G * sizeof(T) + 15) / 16 * 16);
#pragma unroll 1
  for (int i = 4 * threadIdx.x; i < rec.w; i += 4 * kChunkThreads) cp_async<int, 4>(di + i, idx + rec.z + i);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Starts the first two of the steps [s0, s1) (their data must not change before sweep_run)
template <typename T, int G>
__device__ __forceinline__ void sweep_begin(const DevSweep& P, int s0, int s1, const Ring& R, const T* pan0) {
#pragma unroll 1
  for (int k = 0; k < kRingSlots - 1; ++k)
    ring_issue<T, G>(R, k, s0 + k < s1 ? P.step[s0 + k] : make_int4(0, 0, 0, 0), P.idx, pan0);
}

// The steps [s0, s1) by the block, after sweep_begin (TR: with the transposed factors): an
// island's whole range is both substitutions, from its down_ptr the second one.  pan0: the
// panels at the chunk's first lane; v: x and the carried entries at this thread's lane
// (threadIdx.x % G); xs: the teams' fronts.  Ends with a block barrier; every copy it started
// has landed.
template <typename T, int G, int S, bool TR>
__device__ __forceinline__ void sweep_run(const DevSweep& P, int s0, int s1, const Ring& R, T* xs, const T* pan0,
                                          const ChunkVec<T>& v) {
  constexpr int kLg = G == 8 ? 3 : G == 4 ? 2 : G == 2 ? 1 : 0;
  const int n = s1 - s0;
  int slot = 0, free_slot = kRingSlots - 1;
  int4 next = kRingSlots - 1 < n ? P.step[s0 + kRingSlots - 1] : make_int4(0, 0, 0, 0);
  static_assert(kRingSlots == 3, "two steps in flight");
  int ne0 = n > 0 ? P.step[s0].y : 0, ne1 = n > 1 ? P.step[s0 + 1].y : 0;  // their panel entries
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kRingSlots - 2) : "memory");
    __syncthreads();  // step k is in its slot; every thread is done with step k - 1
    ring_issue<T, G>(R, free_slot, next, P.idx, pan0);
    const int ne2 = next.y;
    next = k + kRingSlots < n ? P.step[s0 + k + kRingSlots] : make_int4(0, 0, 0, 0);
    const unsigned char* at = R.base + (size_t)slot * R.slot;
    free_slot = slot;
    slot = slot + 1 == kRingSlots ? 0 : slot + 1;
    // the step's panels start the slot; its index block follows, the step record first
    const T* pan = reinterpret_cast<const T*>(at);
    const int* ib = reinterpret_cast<const int*>(at + ((size_t)ne0 * G * sizeof(T) + 15) / 16 * 16);
    ne0 = ne1;
    ne1 = ne2;
    const int4 q0 = *reinterpret_cast<const int4*>(ib + 4), q1 = *reinterpret_cast<const int4*>(ib + 8);
    const bool up = q0.x != 0;
    const int ls = q0.y, nsolo = q0.z, nbig = q0.w, lteam = q1.x, nteams = q1.y, xstride = q1.z;
    const int4* head = reinterpret_cast<const int4*>(ib + mpf::kStepInts);
    const int busy = nteams << lteam;  // threads of the teams; the others take the solo tasks
    if ((int)threadIdx.x < busy) {
      const int team = 1 << lteam, ti = threadIdx.x >> lteam, tid = threadIdx.x & (team - 1);
      T* x0 = xs + (size_t)ti * xstride * G + threadIdx.x % G;
#pragma unroll 1
      for (int t = ti; t < nbig; t += nteams) {
        const int4 h = head[nsolo + t];
        // a direct step: ib[0] = e0, ib[2] = i0
        const T* us = (q1.w ? pan0 + (size_t)ib[0] * 32 : pan + h.x * G) + threadIdx.x % G;
        const int* xi = q1.w ? P.idx + ib[2] + h.z : ib + h.z;
        const int es = q1.w ? 32 : G;
        if (up) team_subst<T, G, S, true, TR>(h, xi, team, tid, 1 + ti, x0, us, es, v);
        else team_subst<T, G, S, false, TR>(h, xi, team, tid, 1 + ti, x0, us, es, v);
      }
    }
    // solo tasks: thread -> (task, thread r of the lane, lane); a warp whose first task is past
    // the last skips them (the trip count is the same for all its threads)
    const int first = busy < kChunkThreads ? busy : 0;
    const int lsg = ls + kLg, per = (kChunkThreads - first) >> lsg;
    int tw = ((int)(threadIdx.x & ~31u) - first) >> lsg;
    if ((int)threadIdx.x >= first && tw < nsolo) {
      const int split = 1 << ls, r = (threadIdx.x / G) & (split - 1);
      int t = ((int)threadIdx.x - first) >> lsg;
#pragma unroll 1
      do {
        const bool on = t < nsolo;
        const int4 h = head[on ? t : 0];
        const T* p = pan + h.x * G + threadIdx.x % G;
        if (up) solo_subst<T, G, S, true, TR>(on, h, ib, r, split, p, v);
        else solo_subst<T, G, S, false, TR>(on, h, ib, r, split, p, v);
        t += per;
        tw += per;
      } while (tw < nsolo);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

// Both substitutions with the transposed factors of one system (the adjoint's) for a chunk of
// lanes: x in place.  XS: x and the carried entries in shared memory.
template <typename T>
struct SubstChunk {
  DevSweep sw;
  int n;
  long long nnz, sumcbr;
  const T* pan;
  T* cbr;
  T* x;
  int xcap, ccap, scratch, slot;  // as FdChunk
};
template <typename T, int G, bool XS>
__global__ void __launch_bounds__(kChunkThreads, 2) k_subst_chunk(const __grid_constant__ SubstChunk<T> a,
                                                                  const int* __restrict__ group_island) {
  constexpr int LPG = 32 / G, S = XS ? G : 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* const sx = reinterpret_cast<T*>(smem_raw);
  T* const xs = XS ? sx + (size_t)(a.xcap + a.ccap) * G : sx;  // the teams' fronts
  const Ring R{reinterpret_cast<unsigned char*>(xs + (size_t)a.scratch * G), a.slot};
  const int g = blockIdx.x / LPG, lane0 = (blockIdx.x % LPG) * G, l = threadIdx.x % G;
  const int island = group_island ? group_island[g] : 0;
  const T* pan0 = a.pan + at32(g, a.nnz, 0, lane0);
  T* const gx = a.x + at32(g, a.n, 0, lane0 + l);
  const int s0 = a.sw.step_ptr[island], s1 = a.sw.step_ptr[island + 1];
  sweep_begin<T, G>(a.sw, s0, s1, R, pan0);
  if (XS)
    for (int i = threadIdx.x / G; i < a.n; i += kChunkThreads / G) sx[i * G + l] = gx[(size_t)i * 32];
  const ChunkVec<T> v = XS ? ChunkVec<T>{sx + l, sx + (size_t)a.xcap * G + l}
                           : ChunkVec<T>{gx, a.cbr + at32(g, a.sumcbr, 0, lane0 + l)};
  sweep_run<T, G, S, true>(a.sw, s0, s1, R, xs, pan0, v);
  if (XS)
    for (int i = threadIdx.x / G; i < a.n; i += kChunkThreads / G) gx[(size_t)i * 32] = sx[i * G + l];
}

// per-lane max over the block's threads (lane = thread % G), left in red[0 .. G)
template <int G>
__device__ __forceinline__ void chunk_lane_max(double v, double* red) {
#pragma unroll
  for (int o = 16; o >= G; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int ln = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (ln < G) red[warp * G + ln] = v;
  __syncthreads();
  if (threadIdx.x < G) {
    double m = red[threadIdx.x];
    for (int k = 1; k < kChunkThreads / 32; ++k) m = fmax(m, red[k * G + threadIdx.x]);
    red[threadIdx.x] = m;
  }
  __syncthreads();
}

// Fast-decoupled mismatch of the block's lanes, thread = (row slot, lane):
// P = Re(mis)/|V| over PV/PQ, Q = Im(mis)/|V| over PQ (fdpf.h:369-414); returns this thread's
// max over both and writes the side the next half step solves (P, or Q with want_q) to x
template <typename T, int G>
__device__ __forceinline__ double chunk_mismatch_fd(const DevGrid& d, const DevFD& fd, const int* rows, int r0, int r1,
                                                    const LaneOut& o, int g, int lane, T* x, int xs, bool want_q) {
  double lmax = 0.0;
#pragma unroll 1
  for (int r = r0 + threadIdx.x / G; r < r1; r += kChunkThreads / G) {
    const int i = rows[r];
    double2 ib = make_double2(0.0, 0.0);
    const bool touched = row_touched(o, d.y_diag[i]);
    const double2 vi = d.V[at32(g, d.nb, i, lane)];
    const int p0 = d.y_rowptr[i], p1 = d.y_rowptr[i + 1];
    if (touched || d.y_slot) {
      // the row's entries depend on the case
#pragma unroll 1
      for (int p = p0; p < p1; ++p) {
        const double2 y = yentry(d, o, touched, p, g, lane), u = d.V[at32(g, d.nb, d.y_col[p], lane)];
        ib.x += y.x * u.x - y.y * u.y;
        ib.y += y.x * u.y + y.y * u.x;
      }
    } else {
#pragma unroll 1
      for (int p = p0; p < p1; p += 4) {
        int jj[4];
        double2 vv[4], yy[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) jj[u] = p + u < p1 ? d.y_col[p + u] : i;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          vv[u] = jj[u] == i ? vi : d.V[at32(g, d.nb, jj[u], lane)];
          yy[u] = p + u < p1 ? d.y_val[p + u] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (p + u >= p1) break;
          ib.x += yy[u].x * vv[u].x - yy[u].y * vv[u].y;
          ib.y += yy[u].x * vv[u].y + yy[u].y * vv[u].x;
        }
      }
    }
    const double2 s = d.sbus_case ? d.sbus_case[at32(g, d.nb, i, lane)] : d.sbus0[i];
    const double av = sqrt(vi.x * vi.x + vi.y * vi.y);
    const double mr = (vi.x * ib.x + vi.y * ib.y - s.x) / av;
    const double mi = (vi.y * ib.x - vi.x * ib.y - s.y) / av;
    const int2 fv = fd.fdvar[i];
    if (!want_q) x[fv.x * xs] = (T)mr;
    double m = fabs(mr);
    if (mr != mr) m = INFINITY;
    if (fv.y >= 0) {
      if (want_q) x[fv.y * xs] = (T)mi;
      m = fmax(m, fabs(mi));
      if (mi != mi) m = INFINITY;
    }
    lmax = fmax(lmax, finite_or_inf(m));
  }
  return lmax;
}

// The whole fast-decoupled iteration (fdpf.h:450-596) of a chunk of G lanes: mismatch,
// check, then up to max_it iterations of two half steps (forward and backward
// substitution with the stored factors of B' / B'', update, mismatch, check).  Replaces
// a launch per level for each of the four substitutions of an iteration and a host read
// of the "any case running" flag per half step; large
// batches, whose waves of blocks take longer than that, keep the level launches (choose_fd).
// XS: x and the carried entries of the half step in shared memory (else in the systems' arrays)
template <typename T>
struct FdChunk {  // [0]: B' (P half steps), [1]: B'' (Q half steps)
  DevSweep sw[2];
  int n[2];
  long long nnz[2], sumcbr[2];
  const T* pan[2];
  T* cbr[2];
  T* x[2];
  int xcap, ccap, scratch, slot;  // shared memory: entries per lane of x, of the carried
                                  // entries and of the teams' fronts; bytes per ring slot
};
template <typename T, int G, bool XS>
__global__ void __launch_bounds__(kChunkThreads, 1) k_fd_chunk(const __grid_constant__ DevGrid d, DevFD fd,
                                                               const __grid_constant__ FdChunk<T> a, ChunkRows cr,
                                                               int max_it, double tol) {
  constexpr int LPG = 32 / G, S = XS ? G : 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[kChunkThreads / 32 * G];
  __shared__ int st[G];
  __shared__ long long clk[kFdPhases + 1];  // cycles of each phase; when the current one began
  T* const sx = reinterpret_cast<T*>(smem_raw);
  T* const xs = XS ? sx + (size_t)(a.xcap + a.ccap) * G : sx;  // the teams' fronts
  const Ring R{reinterpret_cast<unsigned char*>(xs + (size_t)a.scratch * G), a.slot};
  const int g = blockIdx.x / LPG, lane0 = (blockIdx.x % LPG) * G;
  const int l = threadIdx.x % G, lane = lane0 + l, c = g * 32 + lane;
  const int island = d.group_island ? d.group_island[g] : 0;
  const int r0 = cr.ptr[island], r1 = cr.ptr[island + 1];
  if (threadIdx.x < G) st[threadIdx.x] = d.status[g * 32 + lane0 + threadIdx.x];
  __syncthreads();
  // the mismatch just evaluated decides each running lane (k_check); true while one runs
  auto check = [&](int it, int limit) {
    bool active = false;
    if (threadIdx.x < G && st[threadIdx.x] == ST_RUNNING) {
      const double m = red[threadIdx.x];
      d.maxmis[c] = m;
      d.iters[c] = it;
      int s = ST_RUNNING;
      if (!(m <= DBL_MAX)) s = ST_DIVERGED;
      else if (m < tol) s = ST_CONVERGED;
      else if (it >= limit) s = ST_MAX_ITER;
      else active = true;
      st[threadIdx.x] = s;
    }
    return __syncthreads_or(active) != 0;
  };
  auto vec = [&](int half) {
    if (XS) return ChunkVec<T>{sx + l, sx + (size_t)a.xcap * G + l};
    return ChunkVec<T>{a.x[half] + at32(g, a.n[half], 0, lane), a.cbr[half] + at32(g, a.sumcbr[half], 0, lane)};
  };
  // next: the half step that solves for what this mismatch writes
  auto mismatch = [&](int next) {
    LaneOut o;
    load_outages(d, c, o);
    const ChunkVec<T> v = vec(next);
    chunk_lane_max<G>(chunk_mismatch_fd<T, G>(d, fd, cr.rows, r0, r1, o, g, lane, v.x, S, next == 1), red);
  };
  // a chunk whose lanes were all decided before the solve (padding, cut off) does nothing
  if (!__syncthreads_or(threadIdx.x < G && st[threadIdx.x] == ST_RUNNING)) return;
  auto pan0 = [&](int half) { return a.pan[half] + at32(g, a.nnz[half], 0, lane0); };
  auto begin = [&](int half) {
    const int* sp = a.sw[half].step_ptr + island;
    sweep_begin<T, G>(a.sw[half], sp[0], sp[1], R, pan0(half));
  };
  begin(0);
  auto lap = [&](int phase) {  // the time since the last lap was this phase's
    if (threadIdx.x == 0) {
      const long long now = clock64();
      clk[phase] += now - clk[kFdPhases];
      clk[kFdPhases] = now;
    }
  };
  if (threadIdx.x == 0) {
    for (int k = 0; k < kFdPhases; ++k) clk[k] = 0;
    clk[kFdPhases] = clock64();
  }
  int it = 0, half = 0;
#pragma unroll 1
  for (;;) {
    mismatch(half);
    // after the P half only convergence retires a case (fdpf.h:529-540); the iteration limit
    // is tested after the Q half (and at the start point)
    const bool on = check(it, half == 1 ? INT_MAX : max_it);
    lap(PH_MIS);
    if (!on) break;
    if (half == 0) ++it;
    const ChunkVec<T> v = vec(half);
    const int* sp = a.sw[half].step_ptr + island;
    sweep_run<T, G, S, false>(a.sw[half], sp[0], sp[1], R, xs, pan0(half), v);
    lap(PH_SUBST);
    // the next half step's first panels come in while the voltages are updated
    begin(1 - half);
    if (st[l] == ST_RUNNING)
#pragma unroll 1
      for (int r = r0 + threadIdx.x / G; r < r1; r += kChunkThreads / G) {
        const int i = cr.rows[r];
        const int2 fv = fd.fdvar[i];
        if (half == 1 && fv.y < 0) continue;
        const size_t k = at32(g, d.nb, i, lane);
        const double2 u = d.V[k];
        double mag = sqrt(u.x * u.x + u.y * u.y);
        double ang = vangle(u, d.angle_mode);
        if (half == 0) ang -= (double)v.x[fv.x * S];
        else mag -= (double)v.x[fv.y * S];
        double sn, cs;
        sincos(ang, &sn, &cs);
        d.V[k] = make_double2(mag * cs, mag * sn);
      }
    __syncthreads();
    lap(PH_UPD);
    half = 1 - half;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");  // the copies of a half step not taken
  if (threadIdx.x < G) d.status[c] = st[threadIdx.x];
  if (threadIdx.x == 0) {
    atomicMax(d.it_ptr, it);
    for (int k = 0; k < kFdPhases; ++k)
      atomicAdd(&reinterpret_cast<LoopRecord*>(d.it_ptr)->cycles[k], (unsigned long long)clk[k]);
  }
}

// ---------------------------------------------------------------- Newton on one block
struct DevFactor {
  const int4* step;     // per step: e0, ne, i0, ni
  const int* idx;
  int n;                // steps
};

// Pivots P .. w - 1 of front_rows, one template level per pivot (a loop over 16 pivots is not
// unrolled by the compiler, and a row indexed by a loop variable lives in local memory)
template <typename T, int FR, int LPT, int P>
__device__ __forceinline__ void rows_pivot(int w, int i, bool on, T (&r)[LPT][FR], T (&rhs)[LPT], int* st0) {
  if constexpr (P < FR) {
    if (P >= w) return;
    const bool below = i > P;
#pragma unroll
    for (int k = 0; k < LPT; ++k) {
      T pk = __shfl_sync(0xffffffffu, r[k][P], P, FR);
      if (bad_pivot(pk)) {
        if (i == 0 && on) mark_singular(&st0[k]);
        pk = (T)1;
      }
      const T lip = r[k][P] * ((T)1 / pk);
      if (below) r[k][P] = lip;
#pragma unroll
      for (int q = P + 1; q < FR; ++q) {
        const T u = __shfl_sync(0xffffffffu, r[k][q], P, FR);
        if (below) r[k][q] = r[k][q] - lip * u;
      }
      const T u = __shfl_sync(0xffffffffu, rhs[k], P, FR);
      if (below) rhs[k] = rhs[k] - lip * u;
    }
    rows_pivot<T, FR, LPT, P + 1>(w, i, on, r, rhs, st0);
  }
}

// The partial LU of an assembled front of at most FR rows, and its results, by one warp with
// the rows in registers: thread = (row, group of lanes), each thread its row of LPT lanes;
// pivot rows travel by shuffles.  Same operations per entry as the shared-memory loop.  A
// pivot costs about 220 cycles instead of 900 (300 buses, 257 cases, mixed: factorisation
// 100 -> 60 us).
template <typename T, int G, int FR>
__device__ __forceinline__ void front_rows(int4 h0, int4 h1, const int* rows, int RS, const T* F0, T* cbs0, T* x, T* pan0,
                                           int* st0) {
  constexpr int NG = 32 / FR, LPT = G > NG ? G / NG : 1;
  const int w = h0.z & 0xffff, f = h0.z >> 16, m = f - w;
  const int i = threadIdx.x & (FR - 1), l0 = ((threadIdx.x & 31) / FR) * LPT;
  const bool on = i < f && l0 < G;
  T r[LPT][FR], rhs[LPT];
#pragma unroll
  for (int k = 0; k < LPT; ++k) {
    const T* src = F0 + i * RS * G + l0 + k;
#pragma unroll
    for (int c = 0; c < FR; ++c) r[k][c] = on && c < f ? src[c * G] : (T)0;
    rhs[k] = on ? src[f * G] : (T)0;
  }
  rows_pivot<T, FR, LPT, 0>(w, i, on, r, rhs, st0 + l0);
  if (!on) return;
  const int n = i < w ? f : w;  // panel entries of this row
  T* dst = pan0 + (size_t)(h1.z + (i < w ? i * f : w * f + (i - w) * w)) * 32 + l0;
  T* cd = cbs0 + (h1.x + (i - w) * m - w) * G + l0;
#pragma unroll
  for (int k = 0; k < LPT; ++k) {
#pragma unroll
    for (int c = 0; c < FR; ++c) {
      if (c < n) dst[(size_t)c * 32 + k] = r[k][c];
      else if (c < f && h1.x >= 0) cd[c * G + k] = r[k][c];
    }
    if (i < w) x[rows[i] * G + l0 + k] = rhs[k];
    else if (h1.x >= 0) cbs0[(h1.x + m * m + i - w) * G + l0 + k] = rhs[k];
  }
}

// One front by a team of `team` threads (k_mf_factor's operations), everything it reads in
// shared memory: h0, h1: its header; ib: the step's index block; av: the step's arrowhead
// values; F0: the front; cbs: the contribution blocks; x: the right-hand side, entry i of
// lane l at x[i G + l]; st0: the chunk's statuses, for bad pivots.  Only the panel goes to
// global memory.
template <typename T, int G>
__device__ __forceinline__ void chunk_front(int4 h0, int4 h1, const int* ib, int team, int tid, int bar, const T* av0,
                                            T* F0, T* cbs0, T* x, T* pan0, int* st0) {
  constexpr int V = (int)(16 / sizeof(T)) < G ? (int)(16 / sizeof(T)) : G;
  constexpr int NV = G / V;
  constexpr int U = 4;
  using LV = Lanes<T, V>;
  const int w = h0.z & 0xffff, f = h0.z >> 16, m = f - w, na = h0.y;
  const int slots = team / NV, slot = tid / NV, lv = (tid % NV) * V;
  const int RS = front_stride(f), ncols = f + 1;
  T* F = F0 + lv;
  const int* loc = ib + h0.w;
  const int* rows = loc + na;
  const int* kid = rows + w;
#define FP(r, c) (F + ((r) * RS + (c)) * G)
  {
    LV z;
#pragma unroll
    for (int k = 0; k < V; ++k) z.v[k] = (T)0;
#pragma unroll 1
    for (int i = slot; i < f * RS; i += slots) st<T, V>(F + i * G, z);
  }
  chunk_sync(team, bar);
  {
    const T* av = av0 + h0.x * G + lv;
#pragma unroll 1
    for (int e = slot; e < na; e += slots) st<T, V>(F + loc[e] * G, ld<T, V>(av + e * G));
#pragma unroll 1
    for (int p = slot; p < w; p += slots) st<T, V>(FP(p, f), ld<T, V>(x + rows[p] * G + lv));
  }
  chunk_sync(team, bar);
  // the children's blocks (and right-hand sides), one after the other: siblings may add into
  // the same entries, a child's own places are distinct
#pragma unroll 1
  for (int ci = 0; ci < h1.y; ++ci) {
    const int ne = kid[1];
    const int* to = kid + 2;
    const T* src = cbs0 + kid[0] * G + lv;
#pragma unroll 2
    for (int e = slot; e < ne; e += slots) {
      T* d = F + to[e] * G;
      LV o = ld<T, V>(d);
      const LV v = ld<T, V>(src + e * G);
#pragma unroll
      for (int k = 0; k < V; ++k) o.v[k] += v.v[k];
      st<T, V>(d, o);
    }
    kid = to + ne;
    chunk_sync(team, bar);
  }
  if (team == 32 && f <= (G * sizeof(T) <= 16 ? 16 : 8)) {
    if (f <= 8) front_rows<T, G, 8>(h0, h1, rows, RS, F0, cbs0, x, pan0, st0);
    else if constexpr (G * sizeof(T) <= 16) front_rows<T, G, 16>(h0, h1, rows, RS, F0, cbs0, x, pan0, st0);
    __syncwarp();
    return;
  }
  // row slots x column groups: as many row slots as the front has rows (a power of two)
  int lr = 2;
  while ((1 << lr) < f && (2 << lr) <= slots && lr < 5) ++lr;
  const int rsl = 1 << lr, rs = slot & (rsl - 1), cg = slot >> lr, lc = 31 - __clz(slots >> lr);  // 1 << lc groups
  // right-looking partial LU; with one column group each row's owner writes its scaled L
  // entry back at once, otherwise one pivot later, when no thread reads column p any more
  LV inv_prev;
#pragma unroll 1
  for (int p = 0; p < w; ++p) {
    const LV inv = gather_lanes<T, V>(own_inverse<T, G>(F0[(p * RS + p) * G + (threadIdx.x & 31) % G], tid < G, st0), lv);
    if (lc > 0 && p > 0 && cg == 0)
#pragma unroll 1
      for (int i = p + rs; i < f; i += rsl) {
        LV c = ld<T, V>(FP(i, p - 1));
#pragma unroll
        for (int k = 0; k < V; ++k) c.v[k] *= inv_prev.v[k];
        st<T, V>(FP(i, p - 1), c);
      }
    const int nq = ncols - (p + 1);
    const int q0 = p + 1 + ((nq * cg) >> lc), q1 = p + 1 + ((nq * (cg + 1)) >> lc);
    const T* rp = FP(p, 0);
#pragma unroll 1
    for (int i = p + 1 + rs; i < f; i += rsl) {
      T* ri = FP(i, 0);
      LV lip = ld<T, V>(ri + p * G);
#pragma unroll
      for (int k = 0; k < V; ++k) lip.v[k] *= inv.v[k];
      if (lc == 0) st<T, V>(ri + p * G, lip);
#pragma unroll 1
      for (int q = q0; q < q1; q += U) {
        LV a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (q + u < q1) {
            a[u] = ld<T, V>(rp + (q + u) * G);
            b[u] = ld<T, V>(ri + (q + u) * G);
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (q + u < q1) {
#pragma unroll
            for (int k = 0; k < V; ++k) b[u].v[k] = b[u].v[k] - lip.v[k] * a[u].v[k];
            st<T, V>(ri + (q + u) * G, b[u]);
          }
      }
    }
    inv_prev = inv;
    chunk_sync(team, bar);
  }
  if (lc > 0) {
    if (cg == 0)
#pragma unroll 1
      for (int i = w + rs; i < f; i += rsl) {
        LV c = ld<T, V>(FP(i, w - 1));
#pragma unroll
        for (int k = 0; k < V; ++k) c.v[k] *= inv_prev.v[k];
        st<T, V>(FP(i, w - 1), c);
      }
    chunk_sync(team, bar);
  }
  // panels: rows 0..w-1 all columns, rows w..f-1 the pivot columns; contribution block
  T* pbase = pan0 + (size_t)h1.z * 32 + lv;
  T* cbase = cbs0 + h1.x * G + lv;
#pragma unroll 1
  for (int i = rs; i < f; i += rsl) {
    const T* src = FP(i, 0);
    const int n = i < w ? f : w;
    T* dst = pbase + (size_t)(i < w ? i * f : w * f + (i - w) * w) * 32;
    const int c0 = (n * cg) >> lc, c1 = (n * (cg + 1)) >> lc;
#pragma unroll 2
    for (int q = c0; q < c1; ++q) st<T, V>(dst + (size_t)q * 32, ld<T, V>(src + q * G));
    if (i >= w && h1.x >= 0) {
      const int d0 = (m * cg) >> lc, d1 = (m * (cg + 1)) >> lc;
#pragma unroll 2
      for (int b = d0; b < d1; ++b) st<T, V>(cbase + ((i - w) * m + b) * G, ld<T, V>(src + (w + b) * G));
      if (cg == 0) st<T, V>(cbase + (m * m + i - w) * G, ld<T, V>(FP(i, f)));
    }
  }
#pragma unroll 1
  for (int p = slot; p < w; p += slots) st<T, V>(x + rows[p] * G + lv, ld<T, V>(FP(p, f)));
#undef FP
  chunk_sync(team, bar);
}

// The whole factorisation (with the forward substitution of x) by the block.  a0: the
// arrowhead values at the chunk's first lane; fr: the fronts' shared memory.  Ends with a
// block barrier.
template <typename T, int G>
__device__ __forceinline__ void factor_run(const DevFactor& P, const Ring& R, const T* a0, T* fr, T* cbs, T* x, T* pan0,
                                           int* st0) {
  const int4 none = make_int4(0, 0, 0, 0);
#pragma unroll 1
  for (int k = 0; k < kRingSlots - 1; ++k) ring_issue<T, G>(R, k, k < P.n ? P.step[k] : none, P.idx, a0);
  int slot = 0, free_slot = kRingSlots - 1;
  int4 next = kRingSlots - 1 < P.n ? P.step[kRingSlots - 1] : none;
  int ne0 = P.n > 0 ? P.step[0].y : 0, ne1 = P.n > 1 ? P.step[1].y : 0;
#pragma unroll 1
  for (int k = 0; k < P.n; ++k) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kRingSlots - 2) : "memory");
    __syncthreads();
    ring_issue<T, G>(R, free_slot, next, P.idx, a0);
    const int ne2 = next.y;
    next = k + kRingSlots < P.n ? P.step[k + kRingSlots] : none;
    const unsigned char* at = R.base + (size_t)slot * R.slot;
    free_slot = slot;
    slot = slot + 1 == kRingSlots ? 0 : slot + 1;
    const T* av = reinterpret_cast<const T*>(at);
    const int* ib = reinterpret_cast<const int*>(at + ((size_t)ne0 * G * sizeof(T) + 15) / 16 * 16);
    ne0 = ne1;
    ne1 = ne2;
    const int4 q0 = *reinterpret_cast<const int4*>(ib + 4), q1 = *reinterpret_cast<const int4*>(ib + 8);
    const int nbig = q0.x, nsmall = q0.y, lteam = q0.z, nteams = q0.w, bstride = q1.x, sstride = q1.y;
    const int busy = nteams << lteam;
    const bool big = (int)threadIdx.x < busy;
    // the teams' fronts; the other warps (or all of them after the teams, when these take the
    // whole block) one small front each
#pragma unroll 1
    for (int pass = big ? 0 : 1; pass < 2; ++pass) {
      if (pass == 1 && big) {
        if (busy < kChunkThreads) break;
        if (nsmall > 0) __syncthreads();  // (the whole block: every team is done)
      }
      const int base = pass == 0 || busy >= kChunkThreads ? 0 : busy;
      const int lt = pass == 0 ? lteam : 5, ti = ((int)threadIdx.x - base) >> lt;
      const int nt = pass == 0 ? nteams : (kChunkThreads - base) >> 5;
      const int n = pass == 0 ? nbig : nsmall, t0 = pass == 0 ? 0 : nbig;
      T* F0 = fr + (size_t)(pass == 0 ? ti * bstride : (base > 0 ? nteams * bstride : 0) + ti * sstride) * G;
#pragma unroll 1
      for (int t = ti; t < n; t += nt) {
        const int4* h = reinterpret_cast<const int4*>(ib + mpf::kStepInts + 8 * (t0 + t));
        chunk_front<T, G>(h[0], h[1], ib, 1 << lt, ((int)threadIdx.x - base) & ((1 << lt) - 1), 1 + ti, av, F0, cbs, x,
                          pan0, st0);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
}

// Newton mismatch and Jacobian of the block's lanes (k_mismatch_nr): thread = (row slot,
// lane); F to x (entry i of this lane at x[i G]), the Jacobian to A
template <typename T, int G, bool CTL, bool QL>
__device__ __forceinline__ double chunk_mismatch_nr(const DevGrid& d, const int* rows, int r0, int r1, const LaneOut& o,
                                                    int g, int lane, T* x, T* A) {
  double lmax = 0.0;
#pragma unroll 1
  for (int r = r0 + threadIdx.x / G; r < r1; r += kChunkThreads / G) {
    const int i = rows[r];
    double2 ib = make_double2(0.0, 0.0);
    const int p0 = d.y_rowptr[i], p1 = d.y_rowptr[i + 1], pd = d.y_diag[i];
    const bool touched = row_touched(o, pd);
    const double2 vi = d.V[at32(g, d.nb, i, lane)];
    const bool pvi = QL && still_pv(d, i, g, lane);
    // the next entry's voltage is loaded while this one's entries are formed
    int j = d.y_col[p0], j1 = p0 + 1 < p1 ? d.y_col[p0 + 1] : i;
    double2 v = d.V[at32(g, d.nb, j, lane)];
#pragma unroll 1
    for (int p = p0; p < p1; ++p) {
      const double2 vn = d.V[at32(g, d.nb, j1, lane)];
      const int j2 = p + 2 < p1 ? d.y_col[p + 2] : i;
      const double2 y = yentry<CTL>(d, o, touched, p, g, lane);
      const int4 jp = d.jpos[p];
      ib.x += y.x * v.x - y.y * v.y;
      ib.y += y.x * v.y + y.y * v.x;
      if (j != i && (jp.x >= 0 || jp.y >= 0 || jp.z >= 0 || jp.w >= 0))
        jac_entry(d, A, g, lane, jp, y, v, vi.x, vi.y, 0.0, 0.0, pvi, QL && still_pv(d, j, g, lane));
      v = vn;
      j = j1;
      j1 = j2;
    }
    double2 s = d.sbus_case ? d.sbus_case[at32(g, d.nb, i, lane)] : d.sbus0[i];
    if (QL && !pvi && d.sw_index[i] >= 0) s.y = d.q_fix[at32(g, d.nsw, d.sw_index[i], lane)];
    const double mr = vi.x * ib.x + vi.y * ib.y - s.x;
    const double mi = vi.y * ib.x - vi.x * ib.y - s.y;
    const int2 jv = d.jvar[i];
    x[jv.x * G] = (T)mr;
    double mm = fabs(mr);
    if (jv.y >= 0 && pvi) {
      x[jv.y * G] = (T)0;  // Q of a PV bus is free: its row asks dVm = 0
    } else if (jv.y >= 0) {
      x[jv.y * G] = (T)mi;
      mm = fmax(mm, fabs(mi));
      if (mi != mi) mm = INFINITY;
    }
    if (mr != mr) mm = INFINITY;
    lmax = fmax(lmax, finite_or_inf(mm));
    jac_entry(d, A, g, lane, d.jpos[pd], yentry<CTL>(d, o, touched, pd, g, lane), vi, vi.x, vi.y, ib.x, ib.y, pvi, pvi,
              true);
  }
  return lmax;
}

// Newton's iteration (newtonpf.h:365-523) of a chunk of G lanes by one block.  what =
// NR_ALL: mismatch, check and iterations until no lane runs or max_it are done, in one
// launch; the other values run one part of an iteration (mpf_options.use_graph 0 and 1 time
// the kernel families; x then travels through the LU system's array).  Same operations in
// either form.
enum : int { NR_ALL = 0, NR_FACTOR = 1, NR_SOLVE = 2, NR_UPDATE = 3, NR_MISMATCH = 4 };
template <typename T>
struct NrChunk {
  DevFactor fac;
  DevSweep sw;
  int n, nA;
  long long nnz;
  T* A;
  T* pan;
  T* x;
  // shared memory: x (xcap entries per lane), then for the substitution the teams' fronts
  // (scratch) and its ring (slot bytes per slot), for the factorisation its ring (fslot),
  // the contribution blocks and the fronts (from cbs and fronts, in values per lane)
  int xcap, scratch, slot, fslot, cbs, fronts;
};
template <typename T, int G, bool CTL, bool QL>
__global__ void __launch_bounds__(kChunkThreads, 1) k_nr_chunk(const __grid_constant__ DevGrid d,
                                                               const __grid_constant__ NrChunk<T> a, ChunkRows cr,
                                                               int what, int max_it, double tol) {
  constexpr int LPG = 32 / G;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[kChunkThreads / 32 * G];
  __shared__ int st[G];
  T* const sx = reinterpret_cast<T*>(smem_raw);
  T* const xs = sx + (size_t)a.xcap * G;
  const Ring R{reinterpret_cast<unsigned char*>(xs + (size_t)a.scratch * G), a.slot};
  const int g = blockIdx.x / LPG, lane0 = (blockIdx.x % LPG) * G;
  const int l = threadIdx.x % G, lane = lane0 + l, c = g * 32 + lane;
  const int r0 = cr.ptr[0], r1 = cr.ptr[1];  // one island
  if (threadIdx.x < G) st[threadIdx.x] = d.status[g * 32 + lane0 + threadIdx.x];
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0 && what == NR_UPDATE) atomicAdd(d.it_ptr, 1);
  // a chunk without running lanes does nothing
  if (!__syncthreads_or(threadIdx.x < G && st[threadIdx.x] == ST_RUNNING)) return;
  T* const gx = a.x + at32(g, a.n, 0, lane);
  if (what != NR_ALL && what != NR_MISMATCH) {
    for (int i = threadIdx.x / G; i < a.n; i += kChunkThreads / G) sx[i * G + l] = gx[(size_t)i * 32];
    __syncthreads();
  }
  const T* pan0 = a.pan + at32(g, a.nnz, 0, lane0);
  const int d0 = a.sw.down_ptr[0], d1 = a.sw.step_ptr[1];
  int it = what == NR_MISMATCH ? *d.it_ptr : 0;
#pragma unroll 1
  for (bool first = true;; first = false) {
    if ((what == NR_ALL && !first) || what == NR_FACTOR) {
      factor_run<T, G>(a.fac, Ring{reinterpret_cast<unsigned char*>(xs), a.fslot},
                       a.A + at32(g, a.nA, 0, lane0), xs + a.fronts * G, xs + a.cbs * G, sx,
                       a.pan + at32(g, a.nnz, 0, lane0), st);
    }
    if ((what == NR_ALL && !first) || what == NR_SOLVE) {
      sweep_begin<T, G>(a.sw, d0, d1, R, pan0);
      sweep_run<T, G, G, false>(a.sw, d0, d1, R, xs, pan0, ChunkVec<T>{sx + l, nullptr});
    }
    if ((what == NR_ALL && !first) || what == NR_UPDATE) {
      if (st[l] == ST_RUNNING)
#pragma unroll 1
        for (int r = r0 + threadIdx.x / G; r < r1; r += kChunkThreads / G) {
          const int i = cr.rows[r];
          const int2 jv = d.jvar[i];
          const double dva = (double)sx[jv.x * G + l];
          const double dvm = jv.y >= 0 ? (double)sx[jv.y * G + l] : 0.0;
          const size_t k = at32(g, d.nb, i, lane);
          const double2 v = d.V[k];
          const double mag = sqrt(v.x * v.x + v.y * v.y) - dvm;
          const double ang = vangle(v, d.angle_mode) - dva;
          double sn, cs;
          sincos(ang, &sn, &cs);
          d.V[k] = make_double2(mag * cs, mag * sn);
        }
      ++it;
      __syncthreads();
    }
    if (what == NR_ALL || what == NR_MISMATCH) {
      LaneOut o;
      load_outages(d, c, o);
      chunk_lane_max<G>(chunk_mismatch_nr<T, G, CTL, QL>(d, cr.rows, r0, r1, o, g, lane, sx + l, a.A), red);
      bool active = false;
      if (threadIdx.x < G && st[threadIdx.x] == ST_RUNNING) {  // k_check
        const double m = red[threadIdx.x];
        d.maxmis[c] = m;
        d.iters[c] = it + (d.iter_base ? d.iter_base[c] : 0);
        int s = ST_RUNNING;
        if (!(m <= DBL_MAX)) s = ST_DIVERGED;
        else if (m < tol) s = ST_CONVERGED;
        else if (it >= max_it) s = ST_MAX_ITER;
        else active = true;
        st[threadIdx.x] = s;
      }
      const bool on = __syncthreads_or(active) != 0;
      if (what == NR_MISMATCH && on && threadIdx.x == 0) atomicAdd(d.any_active, 1);
      if (!on) break;
    }
    if (what != NR_ALL) break;
  }
  if (what != NR_ALL && what != NR_UPDATE)
    for (int i = threadIdx.x / G; i < a.n; i += kChunkThreads / G) gx[(size_t)i * 32] = sx[i * G + l];
  if (threadIdx.x < G) d.status[c] = st[threadIdx.x];
  if (what == NR_ALL && threadIdx.x == 0) atomicMax(d.it_ptr, it);
}

}  // namespace mpfk
