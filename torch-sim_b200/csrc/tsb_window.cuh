// Cooperative cell-list search: the candidates of one or several atoms are
// gathered into shared memory once, then tested against each of them.
//
// The atoms' search windows are merged into one box of bins and cut into spans: a
// row of bins within one periodic image along z is a contiguous run of the bin
// order.  32 spans at a time are laid end to end and lane t of a step takes
// candidate t of the run, so lanes stay full whatever the spans' lengths.  A
// candidate is kept when it can lie within the cutoff of one of the atoms, in
// search order, as its shifted FP64 position (x_j + S C, the rounding of a
// one-thread search).  A merged or culled window never changes an atom's hits or
// their order: it only adds or drops candidates beyond the cutoff.
//
// Two shapes share the gathering, one warp each:
//   * one atom per warp (calls too small to fill the GPU): the kept candidates are
//     the atom's hits, 32 of them at a time;
//   * a tile of up to 32 neighbouring atoms per warp (the rest), one lane per atom:
//     a candidate is loaded, shifted and culled once for all of them; every lane
//     then tests the same candidate (one broadcast read) in FP32 against a cutoff
//     widened by the rounding and notes its hits, and the lanes walk their notes
//     together, deciding in FP64.  No divergent loop bounds, and an atom's pairs
//     are summed by its own lane in search order.
//
// Bound: instruction issue (0.6 per cycle and scheduler; the notes' gathers from
// shared memory and the fixed latencies of the test chain fill the rest), not HBM.
// One thread per atom, which this replaces, issued about five times the instructions:
// the lanes of a warp walked bins of different lengths, each bin a bounds load and
// image arithmetic for ~2 atoms.  Measured against it (B200): forces of 540,000
// copper atoms, FP32, 1292 -> 604 us; of 548,000 Kob-Andersen atoms, FP64 with
// stress, 1430 -> 728 us; counting the pairs of 500,000 argon atoms 692 -> 208 us.
// Tried and dropped: one warp per bin (945 us for the argon count: the gathering is
// paid per bin, and 2 atoms share it), one block of four warps per 2 x 2 x 2 bins
// with a ballot per 32 candidates (1245 us), notes walked chunk by chunk in search
// order (295 us, and see SPREAD below).
#pragma once

#include "tsb_search.cuh"

namespace tsb {

constexpr int kWinWarps = 4;  // warps per block

// ------------------------------------------------------------- one warp per atom
// spans of the current run
struct WinSpans {
  double sx[32], sy[32], sz[32];
  int32_t q0[32], pre[32], jx[32], jy[32], jz[32];
};

struct WinSmem : WinSpans {
  static constexpr int kCap = 192;  // kept candidates (more: several chunks)
  double x[kCap], y[kCap], z[kCap];
  int32_t q[kCap];     // slot (bin order)
  int32_t info[kCap];  // species | (unshifted) << 8
  int32_t ix[kCap], iy[kCap], iz[kCap];  // image
};

// a candidate: shifted position, its distance from the atom, tag, slot and span
struct Cand {
  double px, py, pz, dx, dy, dz, d2, w;
  int q, k;
};

// window of one position: bins lo..hi per axis, unbounded on periodic axes
__device__ __forceinline__ void window_of(const SysGeom &G, const double *u, int *lo, int *hi) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double a = floor((u[k] - G.h[k] - G.org[k]) * G.scale[k]);
    double b = floor((u[k] + G.h[k] - G.org[k]) * G.scale[k]);
    if (!G.per[k]) {
      a = fmax(a, 0.0);
      b = fmin(b, (double)(G.nb[k] - 1));
    }
    lo[k] = (int)a;
    hi[k] = (int)b;
  }
}

struct Span {
  int q0, len, ix, iy, iz;
};

// span k of a window lo..hi (nx ny nzs of them, z images fastest)
__device__ __forceinline__ Span span_at(const SysGeom &G, const int64_t *__restrict__ bin_start,
                                        const int *lo, const int *hi, int ny, int iz_lo, int nzs,
                                        int64_t k) {
  Span s;
  const int nb0 = G.nb[0], nb1 = G.nb[1], nb2 = G.nb[2];
  const int r = k <= INT32_MAX ? (int)k / nzs : (int)(k / nzs);
  const int zs = (int)(k - (int64_t)r * nzs);
  const int cx = lo[0] + r / ny, cy = lo[1] + r % ny;
  s.ix = G.per[0] ? floordiv_dev(cx, nb0) : 0;
  s.iy = G.per[1] ? floordiv_dev(cy, nb1) : 0;
  s.iz = iz_lo + zs;
  const int bx = cx - s.ix * nb0, by = cy - s.iy * nb1;
  const int bz0 = max(lo[2], s.iz * nb2) - s.iz * nb2;
  const int bz1 = min(hi[2], s.iz * nb2 + nb2 - 1) - s.iz * nb2;
  const int row = G.bin_base + (bx * nb1 + by) * nb2;
  s.q0 = (int)bin_start[row + bz0];
  s.len = (int)(bin_start[row + bz1 + 1] - s.q0);
  return s;
}

// Gather the candidates of the atom at w that keep(c) takes, put(at, c) each in its
// place and call process(n) on the warp for every full chunk and the last one (also
// when it is empty).  32 spans at a time are laid end to end and lane t of a step takes
// candidate t of the run, so lanes stay full whatever the spans' lengths.
template <class Smem, class K, class T, class F>
__device__ __forceinline__ void window_gather(Smem &S, const SysGeom &G,
                                              const double4 *__restrict__ spos,
                                              const int64_t *__restrict__ bin_start,
                                              const double4 &w, K &&keep_, T &&put,
                                              F &&process) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned le = 0xffffffffu >> (31 - lane), lt = le >> 1;
  if (!(isfinite(w.x) && isfinite(w.y) && isfinite(w.z))) {
    process(0);  // no distance to it is below any cutoff
    return;
  }
  double u[3];
  int lo[3], hi[3];
  frame_coords(G, w.x, w.y, w.z, u);
  window_of(G, u, lo, hi);
  const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1;
  const int iz_lo = G.per[2] ? floordiv_dev(lo[2], G.nb[2]) : 0;
  const int nzs = G.per[2] ? floordiv_dev(hi[2], G.nb[2]) - iz_lo + 1 : (hi[2] >= lo[2]);
  const int64_t n_spans = nx > 0 && ny > 0 && nzs > 0 ? (int64_t)nx * ny * nzs : 0;
  int64_t base = -32;
  int kept = 0, rel = 0, t0 = 0, total = 0;
  int begun = 0;  // spans of the run that start before candidate t0
  bool more = n_spans > 0;
  do {
    while (more && kept <= Smem::kCap - 64) {
      if (t0 >= total) {
        base += 32;
        if (base >= n_spans) {
          more = false;
          break;
        }
        // this lane's span; the non-empty ones are packed into the span table
        Span s{0, 0, 0, 0, 0};
        if (base + lane < n_spans)
          s = span_at(G, bin_start, lo, hi, ny, iz_lo, nzs, base + lane);
        int inc = s.len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(full, inc, o);
          if (lane >= o) inc += t;
        }
        total = __shfl_sync(full, inc, 31);
        const unsigned some = __ballot_sync(full, s.len > 0);
        __syncwarp();  // the table's last readers are done
        if (s.len > 0) {
          const int r = __popc(some & lt);
          S.q0[r] = s.q0;
          S.pre[r] = inc - s.len;
          S.sx[r] = s.ix * G.cell[0] + s.iy * G.cell[3] + s.iz * G.cell[6];
          S.sy[r] = s.ix * G.cell[1] + s.iy * G.cell[4] + s.iz * G.cell[7];
          S.sz[r] = s.ix * G.cell[2] + s.iy * G.cell[5] + s.iz * G.cell[8];
          S.jx[r] = s.ix;
          S.jy[r] = s.iy;
          S.jz[r] = s.iz;
        }
        __syncwarp();
        rel = lane < __popc(some) ? S.pre[lane] : INT32_MAX;
        begun = 0;
        t0 = 0;
        continue;
      }
      // two steps of 32 at once, so that both loads are in flight
      double4 o[2];
      int k[2], q[2];
      bool in[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int tb = t0 + 32 * h, t = tb + lane;
        const unsigned d = (unsigned)(rel - tb);
        const unsigned starts = __reduce_or_sync(full, d < 32u ? 1u << d : 0u);
        k[h] = begun + __popc(starts & le) - 1;
        begun += __popc(starts);
        in[h] = t < total;
        q[h] = 0;
        o[h] = make_double4(0.0, 0.0, 0.0, 0.0);
        if (in[h]) {
          q[h] = S.q0[k[h]] + (t - S.pre[k[h]]);
          o[h] = spos[q[h]];
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Cand c{};
        if (in[h]) {
          c.px = o[h].x + S.sx[k[h]];
          c.py = o[h].y + S.sy[k[h]];
          c.pz = o[h].z + S.sz[k[h]];
          c.dx = c.px - w.x;
          c.dy = c.py - w.y;
          c.dz = c.pz - w.z;
          c.d2 = c.dx * c.dx + c.dy * c.dy + c.dz * c.dz;
          c.w = o[h].w;
          c.q = q[h];
          c.k = k[h];
          in[h] = keep_(c);
        }
        const unsigned keep = __ballot_sync(full, in[h]);
        if (in[h]) put(kept + __popc(keep & lt), c);
        kept += __popc(keep);
      }
      t0 += 64;
    }
    __syncwarp();
    process(kept);
    __syncwarp();
    kept = 0;
  } while (more);
}

// every candidate within the cutoff (and its rounding), with all that is known of it
template <class F>
__device__ __forceinline__ void window_gather(WinSmem &S, const SysGeom &G,
                                              const double4 *__restrict__ spos,
                                              const int64_t *__restrict__ bin_start,
                                              const double4 &w, double cutoff, F &&process) {
  const double reach2 = cutoff * cutoff * (1.0 + 1e-12);
  window_gather(
      S, G, spos, bin_start, w, [&](const Cand &c) { return c.d2 < reach2; },
      [&](int at, const Cand &c) {
        S.x[at] = c.px;
        S.y[at] = c.py;
        S.z[at] = c.pz;
        S.q[at] = c.q;
        const int ii = S.jx[c.k], jj = S.jy[c.k], ll = S.jz[c.k];
        S.info[at] = min(max(tag_species(c.w), 0), 255) | ((ii | jj | ll) == 0 ? 256 : 0);
        S.ix[at] = ii;
        S.iy[at] = jj;
        S.iz[at] = ll;
      },
      process);
}

// ------------------------------------------------------------ a tile per warp
constexpr int kTileNotes = 64;    // hits a lane notes before the warp walks them
constexpr int kTileStride = 36;   // bytes between a lane's notes (no bank conflicts
                                  // along either index)

// SHIFT keeps each candidate's image minus its integer wrap (neighbour lists)
template <bool SHIFT>
struct TileSmem {
  // kept candidates (more: several chunks); six (SHIFT: five) blocks of four warps
  // fit an SM
  static constexpr int kCap = SHIFT ? 128 : 132;
  double x[kCap], y[kCap], z[kCap];
  // relative to the tile's centre, padded to whole groups of four by far ones
  alignas(16) float fx[kCap];
  alignas(16) float fy[kCap];
  alignas(16) float fz[kCap];
  int32_t j[kCap];  // atom | (unshifted) << 30
  int32_t shift[SHIFT ? 3 : 1][SHIFT ? kCap : 1];
  uint8_t spec[SHIFT ? 8 : kCap];
  uint8_t note[kTileNotes * kTileStride];
  double sx[32], sy[32], sz[32];  // spans of the current run
  int32_t q0[32], pre[32], jx[32], jy[32], jz[32];
};

// A tile: slots order[off .. off + m), m <= 32, of system sys.  The atoms of a system
// are put in column order (tsb_bins.cu): columns of 2 x 2 rows of bins, along z within
// a column, so that 32 in a row fill a compact box.
struct Tile {
  int32_t off, m, sys;
};

// rows of bins per column and axis
__device__ __forceinline__ void column_dims(const SysGeom &G, int &gx, int &gy) {
  const float a = (float)G.count / (float)G.nbins;
  gy = a < 16.0f && G.nb[1] > 1 ? 2 : 1;
  gx = a < 8.0f && G.nb[0] > 1 ? 2 : 1;
}

// blocks of the persistent tile kernels: what their shared memory lets an SM hold
template <class K>
inline unsigned tile_grid(K kernel, size_t bytes) {
  int dev = 0, n_sm = 148, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 32 * kWinWarps, bytes) !=
          cudaSuccess || per < 1)
    per = 1;
  return (unsigned)(per * n_sm);
}

// The warp's next tile, or -1: tiles differ in cost (a small cell's window takes many
// short spans), so warps draw them one by one; the index is drawn a tile ahead.
struct TileQueue {
  int next;
  __device__ __forceinline__ explicit TileQueue(const TileList &t) { next = draw(t); }
  __device__ __forceinline__ int draw(const TileList &t) {
    int k = 0;
    if ((threadIdx.x & 31) == 0) k = atomicAdd(t.n_tiles + 1, 1);
    return k;
  }
  __device__ __forceinline__ int take(const TileList &t, int n) {
    const int k = __shfl_sync(0xffffffffu, next, 0);
    if (k >= n) return -1;
    next = draw(t);
    return k;
  }
};

// May these atoms share a window?  Only positions that the wrap brought into (or
// left near) the cell: a clamped wrap of an enormous coordinate would stretch the
// merged box over every image in between, a NaN would spoil the centre.
__device__ __forceinline__ bool window_mergeable(const SysGeom &G, const double4 &w,
                                                 const double *u) {
  bool ok = isfinite(w.x) && isfinite(w.y) && isfinite(w.z);
#pragma unroll
  for (int k = 0; k < 3; ++k) ok = ok && (!G.per[k] || fabs(u[k]) < 4.0);
  return ok;
}

// minimum / maximum over the warp of a finite FP32 value (as ordered integers)
__device__ __forceinline__ float warp_max_f(float v) {
  const int b = __float_as_int(v);
  const int k = __reduce_max_sync(0xffffffffu, b ^ ((b >> 31) & 0x7fffffff));
  return __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
}

// One lane's atom of a tile.
struct TileAtom {
  double4 w;   // wrapped position, tag
  float fx, fy, fz;  // relative to the tile's centre; out of reach without an atom
  int i;             // atom | 1 << 30: its own unshifted image in TileSmem::j
  bool have;
  bool wrapped;      // in or near the cell, so its window holds its own bin
};

// The atoms of a tile (together when they may share a window, else one by one):
// begin(A) once per batch with the lanes' atoms, process(A, kept, pre2) for every chunk
// of kept candidates (pre2: the widened cutoff^2; as far below the cutoff^2 a pair is
// surely inside), end(A) after the last.
// wraps: the integer wraps by slot, for SHIFT.
// SPREAD takes the spans in a scattered order (a fixed one, by the window's shape):
// in search order a chunk is a slab of the window, near some of the atoms and out of
// reach of the rest, and the lanes that walk their notes wait for the longest (3-4
// times the mean).  For passes whose result does not depend on the order.
template <bool SPREAD, bool SHIFT, class B, class F, class E>
__device__ __forceinline__ void tile_gather(TileSmem<SHIFT> &S, const BinData &b, const Tile &T,
                                            const int32_t *__restrict__ order,
                                            const int4 *__restrict__ wraps, double cutoff,
                                            B &&begin, F &&process, E &&end) {
  const SysGeom &G = b.geom[T.sys];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned le = 0xffffffffu >> (31 - lane), lt = le >> 1;
  const double4 *__restrict__ spos = b.spos;
  const int64_t *__restrict__ bin_start = b.bin_start;
  for (int a0 = 0; a0 < T.m;) {
    int m = T.m - a0;
    TileAtom A;
    A.w = make_double4(0.0, 0.0, 0.0, 0.0);
    if (lane < m) A.w = spos[order[T.off + a0 + lane]];
    A.i = tag_atom(A.w.w) | 1 << 30;
    double u[3];
    frame_coords(G, A.w.x, A.w.y, A.w.z, u);
    A.wrapped = window_mergeable(G, A.w, u);
    if (!__all_sync(full, lane >= m || A.wrapped)) m = 1;
    A.have = lane < m;
    int lo[3], hi[3];
    window_of(G, u, lo, hi);
    const bool lost = m == 1 && !(isfinite(A.w.x) && isfinite(A.w.y) && isfinite(A.w.z));
    const bool any = !__shfl_sync(full, (int)lost, 0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = __reduce_min_sync(full, A.have ? lo[k] : INT32_MAX);
      hi[k] = __reduce_max_sync(full, A.have ? hi[k] : INT32_MIN);
    }
    // the atoms' box around the first of them (FP32 extents, rounded outwards)
    const double cx = __shfl_sync(full, A.w.x, 0), cy = __shfl_sync(full, A.w.y, 0),
                 cz = __shfl_sync(full, A.w.z, 0);
    A.fx = A.fy = A.fz = 0.0f;
    if (A.have) {
      A.fx = (float)(A.w.x - cx);
      A.fy = (float)(A.w.y - cy);
      A.fz = (float)(A.w.z - cz);
    }
    const float bx1 = warp_max_f(A.fx), bx0 = -warp_max_f(-A.fx);
    const float by1 = warp_max_f(A.fy), by0 = -warp_max_f(-A.fy);
    const float bz1 = warp_max_f(A.fz), bz0 = -warp_max_f(-A.fz);
    // a kept candidate lies within reach of the box, so every coordinate below is
    // at most M: two of them rounded to FP32, their difference and the sum of
    // squares put r^2 within 11 * 2^-24 M^2 of the FP64 value
    const float M = (float)cutoff + fmaxf(fmaxf(bx1, -bx0), fmaxf(fmaxf(by1, -by0),
                                                                  fmaxf(bz1, -bz0)));
    const float pre2 = __double2float_ru(cutoff * cutoff + (double)(M * M) * 0x1p-19);
    if (!A.have) A.fx = -1e18f;  // no candidate is near
    begin(A);
    const int ny = hi[1] - lo[1] + 1, nx = hi[0] - lo[0] + 1;
    const int iz_lo = G.per[2] ? floordiv_dev(lo[2], G.nb[2]) : 0;
    const int nzs = G.per[2] ? floordiv_dev(hi[2], G.nb[2]) - iz_lo + 1 : (hi[2] >= lo[2]);
    const int64_t n_spans =
        any && nx > 0 && ny > 0 && nzs > 0 ? (int64_t)nx * ny * nzs : 0;
    unsigned stride = 1;
    const bool spread = SPREAD && n_spans > 8 && n_spans < (1 << 15);
    if (spread) {
      // the first step >= 0.38 n without a common divisor
      const int s0 = (int)(0.38f * (float)n_spans) + lane;
      int x = (int)n_spans, y = s0;
      while (y) {
        const int r = x % y;
        x = y;
        y = r;
      }
      const unsigned ok = __ballot_sync(full, x == 1);
      if (ok) stride = (unsigned)__shfl_sync(full, s0, __ffs(ok) - 1);
    }
    int64_t base = -32;
    int kept = 0, rel = 0, t0 = 0, total = 0;
    int begun = 0;  // spans of the run that start before candidate t0
    bool more = n_spans > 0;
    while (more) {
      while (kept <= TileSmem<SHIFT>::kCap - 64) {
        if (t0 >= total) {
          base += 32;
          if (base >= n_spans) {
            more = false;
            break;
          }
          // this lane's span; the non-empty ones are packed into the span table
          Span s{0, 0, 0, 0, 0};
          if (base + lane < n_spans)
            s = span_at(G, bin_start, lo, hi, ny, iz_lo, nzs,
                        spread ? (unsigned)(base + lane) * stride % (unsigned)n_spans
                               : base + lane);
          int inc = s.len;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(full, inc, o);
            if (lane >= o) inc += t;
          }
          total = __shfl_sync(full, inc, 31);
          const unsigned some = __ballot_sync(full, s.len > 0);
          __syncwarp();  // the table's last readers are done
          if (s.len > 0) {
            const int r = __popc(some & lt);
            S.q0[r] = s.q0;
            S.pre[r] = inc - s.len;
            S.sx[r] = s.ix * G.cell[0] + s.iy * G.cell[3] + s.iz * G.cell[6];
            S.sy[r] = s.ix * G.cell[1] + s.iy * G.cell[4] + s.iz * G.cell[7];
            S.sz[r] = s.ix * G.cell[2] + s.iy * G.cell[5] + s.iz * G.cell[8];
            S.jx[r] = s.ix;
            S.jy[r] = s.iy;
            S.jz[r] = s.iz;
          }
          __syncwarp();
          rel = lane < __popc(some) ? S.pre[lane] : INT32_MAX;
          begun = 0;
          t0 = 0;
          continue;
        }
        // two steps of 32 at once, so that both loads are in flight
        double4 o[2];
        int4 wr[2];
        int k[2];
        bool in[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int tb = t0 + 32 * h, t = tb + lane;
          const unsigned d = (unsigned)(rel - tb);
          const unsigned starts = __reduce_or_sync(full, d < 32u ? 1u << d : 0u);
          k[h] = begun + __popc(starts & le) - 1;
          begun += __popc(starts);
          in[h] = t < total;
          o[h] = make_double4(0.0, 0.0, 0.0, 0.0);
          wr[h] = make_int4(0, 0, 0, 0);
          if (in[h]) {
            const int q = S.q0[k[h]] + (t - S.pre[k[h]]);
            o[h] = spos[q];
            if constexpr (SHIFT) wr[h] = wraps[q];
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          double px = 0.0, py = 0.0, pz = 0.0;
          float fx = 0.f, fy = 0.f, fz = 0.f;
          if (in[h]) {
            px = o[h].x + S.sx[k[h]];
            py = o[h].y + S.sy[k[h]];
            pz = o[h].z + S.sz[k[h]];
            fx = (float)(px - cx);
            fy = (float)(py - cy);
            fz = (float)(pz - cz);
            // distance to the box, from above by the slack of pre2
            const float ex = fmaxf(fmaxf(bx0 - fx, fx - bx1), 0.0f);
            const float ey = fmaxf(fmaxf(by0 - fy, fy - by1), 0.0f);
            const float ez = fmaxf(fmaxf(bz0 - fz, fz - bz1), 0.0f);
            in[h] = ex * ex + ey * ey + ez * ez < pre2;
          }
          const unsigned keep = __ballot_sync(full, in[h]);
          if (in[h]) {
            const int at = kept + __popc(keep & lt), kk = k[h];
            S.x[at] = px;
            S.y[at] = py;
            S.z[at] = pz;
            const int ii = S.jx[kk], jj = S.jy[kk], ll = S.jz[kk], j = tag_atom(o[h].w);
            S.fx[at] = fx;
            S.fy[at] = fy;
            S.fz[at] = fz;
            S.j[at] = j | ((ii | jj | ll) == 0 ? 1 << 30 : 0);
            if constexpr (SHIFT) {
              // shifts valid for the unwrapped positions (torch_nl.py:214), up to the
              // atom's own wrap
              S.shift[0][at] = ii - wr[h].x;
              S.shift[1][at] = jj - wr[h].y;
              S.shift[2][at] = ll - wr[h].z;
            } else {
              S.spec[at] = (uint8_t)min(max(tag_species(o[h].w), 0), 255);
            }
          }
          kept += __popc(keep);
        }
        t0 += 64;
      }
      if (lane < (-kept & 3)) {  // pad to a whole group of four
        S.fx[kept + lane] = 3e18f;
        S.fy[kept + lane] = S.fz[kept + lane] = 0.0f;
      }
      __syncwarp();
      process(A, kept, pre2);
      __syncwarp();
      kept = 0;
    }
    end(A);
    a0 += m;
  }
}

// two FP32 sums / fused products at once (each rounded on its own)
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}

// Every lane tests candidates t0.. against its atom and notes the near ones, four
// candidates per step (one broadcast read per axis); the scan stops at the end or
// when a lane's notes are nearly full.  Returns the next candidate; n_notes is the
// lane's count.  COUNT adds the candidates that are inside whatever the rounding
// (below sure2) to n_sure and notes only the others.
template <bool COUNT, bool SHIFT>
__device__ __forceinline__ int tile_scan(TileSmem<SHIFT> &S, const TileAtom &A, int t0, int kept,
                                         float pre2, int &n_notes, float sure2, int &n_sure) {
  const int lane = threadIdx.x & 31;
  uint8_t *note = S.note + lane, *const nearly = note + (kTileNotes - 4) * kTileStride;
  const unsigned long long ax = pack2(-A.fx, -A.fx), ay = pack2(-A.fy, -A.fy),
                           az = pack2(-A.fz, -A.fz);
  int t = t0;
  for (; t < kept; t += 4) {
    if (__any_sync(0xffffffffu, note > nearly)) break;
    const ulonglong2 X = *(const ulonglong2 *)(S.fx + t), Y = *(const ulonglong2 *)(S.fy + t),
                     Z = *(const ulonglong2 *)(S.fz + t);
    const unsigned long long dx0 = add2(X.x, ax), dy0 = add2(Y.x, ay), dz0 = add2(Z.x, az);
    const unsigned long long dx1 = add2(X.y, ax), dy1 = add2(Y.y, ay), dz1 = add2(Z.y, az);
    const float2 r0 = unpack2(fma2(dz0, dz0, fma2(dy0, dy0, mul2(dx0, dx0))));
    const float2 r1 = unpack2(fma2(dz1, dz1, fma2(dy1, dy1, mul2(dx1, dx1))));
    const float r2[4] = {r0.x, r0.y, r1.x, r1.y};
    if constexpr (COUNT) {
      bool band = false;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        n_sure += r2[k] < sure2;
        band = band || (r2[k] >= sure2 && r2[k] < pre2);
      }
      if (!band) continue;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (r2[k] < pre2 && (!COUNT || r2[k] >= sure2)) {
        *note = (uint8_t)(t + k);
        note += kTileStride;
      }
  }
  n_notes = (int)(note - (S.note + lane)) / kTileStride;
  __syncwarp();
  return t;
}

// Sums NV (a power of two, at most 32) values per lane over the warp by
// exchanging halves: afterwards lane l holds the total of value
// l / (32 / NV) (32 / NV lanes hold the same one), in 2 NV - 2 + log2(32 / NV)
// exchanges instead of 5 NV.
template <int NV, class T>
__device__ __forceinline__ T warp_multi_sum(T *v) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int n = NV / 2; n >= 1; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int k = 0; k < n; ++k) {
      const T send = up ? v[k] : v[k + n];
      const T keep = up ? v[k + n] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  T t = v[0];
  for (; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

}  // namespace tsb
