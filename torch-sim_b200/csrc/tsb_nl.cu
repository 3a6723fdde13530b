// Neighbour-list construction (drop-in for torch_nl_linked_cell,
// torch_sim/neighbors/torch_nl.py:156-215).  Two passes over a cell-list
// search: count per atom -> exclusive scan -> fill, so the output is grouped by
// the central atom i in ascending order and deterministic (within an atom: the
// order of the search's bins, ascending atom index inside a bin).
#include "tsb_window.cuh"

namespace tsb {

// full_to_half_list rule (pair_potential.py:86-127): keep i < j; for i == j keep
// the copy whose first non-zero shift component is positive.
__device__ inline bool keep_half(int i, int j, int sx, int sy, int sz) {
  if (i != j) return i < j;
  int first = sx != 0 ? sx : (sy != 0 ? sy : sz);
  return first > 0;
}

// Two passes over the gathered candidates (tsb_window.cuh): FILL = false counts
// each atom's pairs, FILL = true writes them.  Hits are written 32 at a time, so an
// atom's rows leave as contiguous stores (one thread per atom wrote its 36-56 bytes
// per pair to rows of its own: 2.77 ms on the 500,000-atom list, now 0.75 ms; the
// bytes alone take 0.2 ms).  With `packed` the second mapping row starts at the pair
// count, read from off[n], and nothing is written unless every pair fits.
template <class P>
struct NlOut {
  const int64_t *off;
  int64_t cap;
  int packed;
  int64_t *mapping;
  int64_t stride;
  int64_t *system_mapping;
  P *shifts;
};

// one atom's side of a pass: which of a warp's candidates are its pairs, and where
// they go
template <class P, bool FILL>
struct NlAtom {
  int i, s;
  int W0, W1, W2;
  int64_t o;  // FILL: next row; else pairs so far

  // pairs among the lanes' candidates (slot q, image sx, sy, sz; `in`: within the
  // cutoff and not the atom itself)
  __device__ __forceinline__ void take(const BinData &b, bool in, int q, int sx, int sy, int sz,
                                       bool half, const NlOut<P> &out, P *buf) {
    const int lane = threadIdx.x & 31;
    int j = 0, fx = 0, fy = 0, fz = 0;
    if ((FILL || half) && in) {
      // shifts valid for the unwrapped positions (torch_nl.py:214)
      j = b.sidx[q];
      const int32_t *W = b.wrap + 3 * (int64_t)j;
      fx = sx + W0 - W[0];
      fy = sy + W1 - W[1];
      fz = sz + W2 - W[2];
      if (half) in = keep_half(i, j, fx, fy, fz);
    }
    const unsigned m = __ballot_sync(0xffffffffu, in);
    const int c = __popc(m);
    if constexpr (FILL) {
      const int k = __popc(m & ((1u << lane) - 1u));
      if (in) {
        const int64_t r = o + k;
        if (r < out.cap) {
          out.mapping[r] = i;
          out.mapping[out.stride + r] = j;
          out.system_mapping[r] = s;
        }
        buf[3 * k] = (P)fx;
        buf[3 * k + 1] = (P)fy;
        buf[3 * k + 2] = (P)fz;
      }
      __syncwarp();
      const int n3 = 3 * (int)max((int64_t)0, min((int64_t)c, out.cap - o));
      for (int e = lane; e < n3; e += 32) out.shifts[3 * o + e] = buf[e];
      __syncwarp();
    }
    o += c;
  }
};

template <class P, bool FILL>
__device__ __forceinline__ NlAtom<P, FILL> nl_atom(const BinData &b, int i, int s, int64_t o) {
  const int32_t *W = b.wrap + 3 * (int64_t)i;
  return NlAtom<P, FILL>{i, s, W[0], W[1], W[2], o};
}

// small lists: one warp per atom
template <class P, bool FILL>
__global__ void __launch_bounds__(32 * kWinWarps)
    k_nl_warp(BinData b, int64_t n, double cutoff, int flags, int32_t *cnt, NlOut<P> out) {
  __shared__ WinSmem win[kWinWarps];
  __shared__ P buf[FILL ? kWinWarps : 1][FILL ? 96 : 1];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t p = (int64_t)blockIdx.x * kWinWarps + wid;
  if (p >= n) return;
  if (FILL && out.packed) {
    out.stride = out.off[n];
    if (out.stride > out.cap) return;
  }
  const double4 w = b.spos[p];
  const int i = tag_atom(w.w), s = b.sys_of[i];
  const bool self = flags & TSB_NL_SELF_INTERACTION, half = flags & TSB_NL_HALF;
  const double rc2 = cutoff * cutoff;
  WinSmem &S = win[wid];
  NlAtom<P, FILL> A = nl_atom<P, FILL>(b, i, s, FILL ? out.off[i] : 0);
  window_gather(S, b.geom[s], b.spos, b.bin_start, w, cutoff, [&](int kept) {
    for (int t0 = 0; t0 < kept; t0 += 32) {
      const int t = t0 + lane;
      bool in = t < kept;
      if (in) {
        const double dx = S.x[t] - w.x, dy = S.y[t] - w.y, dz = S.z[t] - w.z;
        in = dx * dx + dy * dy + dz * dz < rc2 &&
             (self || !(S.q[t] == p && (S.info[t] & 256)));
      }
      const int u = in ? t : 0;
      A.take(b, in, S.q[u], S.ix[u], S.iy[u], S.iz[u], half, out, buf[FILL ? wid : 0]);
    }
  });
  if (!FILL && lane == 0) cnt[i] = (int32_t)A.o;
}

// large lists: one warp per tile.  Counting a full list needs FP64 only for
// candidates within the FP32 rounding of the cutoff.  Filling (and half lists), the
// warp takes all lanes' notes end to end: one note per lane decides in FP64, and an
// atom's pairs leave as contiguous rows.
template <class P, bool FILL, bool HALF>
__global__ void __launch_bounds__(32 * kWinWarps, FILL || HALF ? 5 : 6)
    k_nl_tile(BinData b, int64_t n, TileList tl, const int4 *__restrict__ wraps, double cutoff,
              int flags, int32_t *cnt, NlOut<P> out) {
  constexpr bool ROWS = FILL || HALF;
  struct Warp {
    TileSmem<ROWS> tile;
    // lanes with notes, by rank: the notes before theirs, the lane, its pairs so far
    int32_t pre[ROWS ? 32 : 1], got[ROWS ? 32 : 1];
    uint8_t own[ROWS ? 32 : 8];
    // by lane: wrap and next row of its atom
    int32_t W[3][ROWS ? 32 : 1];
    int64_t row[FILL ? 32 : 1];
  };
  __shared__ Warp smem[kWinWarps];
  if (FILL && out.packed) {
    out.stride = out.off[n];
    if (out.stride > out.cap) return;
  }
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned le = 0xffffffffu >> (31 - lane), lt = le >> 1;
  const bool self = flags & TSB_NL_SELF_INTERACTION;
  const double rc2 = cutoff * cutoff;
  Warp &me = smem[wid];
  TileSmem<ROWS> &S = me.tile;
  const int nt = *tl.n_tiles;
  TileQueue queue(tl);
  for (int g; (g = queue.take(tl, nt)) >= 0;) {
    const Tile T = tl.tiles[g];
    const int s = T.sys;
    int64_t at = 0;  // of the lane's atom: FILL: next row; else its count
    tile_gather<!ROWS>(
        S, b, T, tl.order, wraps, cutoff,
        [&](const TileAtom &A) {
          at = 0;
          if constexpr (ROWS) {
            const int i = tag_atom(A.w.w);
            if (FILL && A.have) at = out.off[i];
            const int32_t *W = b.wrap + 3 * (int64_t)i;
            __syncwarp();
            for (int k = 0; k < 3; ++k) me.W[k][lane] = A.have ? W[k] : 0;
          }
        },
        [&](const TileAtom &A, int kept, float pre2) {
          const float sure2 = __double2float_rd(rc2 - ((double)pre2 - rc2));
          for (int t0 = 0; t0 < kept;) {
            int nn, sure = 0;
            t0 = tile_scan<!ROWS>(S, A, t0, kept, pre2, nn, sure2, sure);
            if constexpr (!ROWS) {
              at += sure;
              for (int k = 0; k < nn; ++k) {
                const int t = S.note[k * kTileStride + lane];
                const double dx = S.x[t] - A.w.x, dy = S.y[t] - A.w.y, dz = S.z[t] - A.w.z;
                at += dx * dx + dy * dy + dz * dz < rc2;
              }
            } else {
              int inc = nn;
#pragma unroll
              for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(full, inc, o);
                if (lane >= o) inc += u;
              }
              const int total = __shfl_sync(full, inc, 31);
              const unsigned some = __ballot_sync(full, nn > 0);
              const int rank = __popc(some & lt);
              if (nn > 0) {
                me.own[rank] = (uint8_t)lane;
                me.pre[rank] = inc - nn;
                me.got[rank] = 0;
              }
              if constexpr (FILL) me.row[lane] = at;
              __syncwarp();
              const int rel = lane < __popc(some) ? me.pre[lane] : INT32_MAX;
              int begun = 0, carry = 0;  // carry: pairs of the atom the last step ended in
              for (int e0 = 0; e0 < total; e0 += 32) {
                const int e = e0 + lane;
                const unsigned d = (unsigned)(rel - e0);
                const unsigned starts = __reduce_or_sync(full, d < 32u ? 1u << d : 0u);
                const int r = begun + __popc(starts & le) - 1;
                begun += __popc(starts);
                const int a = me.own[r];
                const double wx = __shfl_sync(full, A.w.x, a), wy = __shfl_sync(full, A.w.y, a),
                             wz = __shfl_sync(full, A.w.z, a);
                const int ai = __shfl_sync(full, A.i, a);
                bool in = e < total;
                const int t = in ? S.note[(e - me.pre[r]) * kTileStride + a] : 0;
                const int j = S.j[t];
                const double dx = S.x[t] - wx, dy = S.y[t] - wy, dz = S.z[t] - wz;
                const double d2 = dx * dx + dy * dy + dz * dz;
                in = in && d2 < rc2 && (self || !(d2 == 0.0 && j == ai));
                const int i0 = ai & ~(1 << 30), j0 = j & ~(1 << 30);
                const int fx = S.shift[0][t] + me.W[0][a], fy = S.shift[1][t] + me.W[1][a],
                          fz = S.shift[2][t] + me.W[2][a];
                if (HALF) in = in && keep_half(i0, j0, fx, fy, fz);
                // place among the atom's pairs: those since its first note
                const unsigned m = __ballot_sync(full, in);
                const unsigned mine = starts & le;
                const int first = mine ? 31 - __clz(mine) : 0;
                const int k = __popc(m & lt & ~((1u << first) - 1u)) + (mine ? 0 : carry);
                if (in) {
                  // the atom's last pair of this step leaves the count
                  const unsigned later = starts & ~le;
                  const unsigned rest =
                      m & ~le & (later ? (1u << (__ffs(later) - 1)) - 1u : full);
                  if (!rest) me.got[r] = k + 1;
                  if constexpr (FILL) {
                    const int64_t row = me.row[a] + k;
                    if (row < out.cap) {
                      // written once, not read here: the positions stay in L2
                      __stcs((long long *)out.mapping + row, (long long)i0);
                      __stcs((long long *)out.mapping + out.stride + row, (long long)j0);
                      __stcs((long long *)out.system_mapping + row, (long long)s);
                      P *sh = out.shifts + 3 * row;
                      __stcs(sh, (P)fx);
                      __stcs(sh + 1, (P)fy);
                      __stcs(sh + 2, (P)fz);
                    }
                  }
                }
                const int lf = starts ? 31 - __clz(starts) : 0;
                carry = __popc(m & ~((1u << lf) - 1u)) + (starts ? 0 : carry);
              }
              __syncwarp();
              if (nn > 0) at += me.got[rank];
            }
            __syncwarp();
          }
        },
        [&](const TileAtom &A) {
          // (the sure ones of a wrapped atom include its own unshifted image)
          if (!FILL && A.have)
            cnt[tag_atom(A.w.w)] = (int32_t)(at - (!ROWS && !self && A.wrapped));
        });
  }
}

// integer wraps by slot, so that a run of candidates reads them as it reads the
// positions
__global__ void k_nl_wraps(const int32_t *sidx, const int32_t *wrap, int64_t n, int4 *wraps) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int32_t *W = wrap + 3 * (int64_t)sidx[p];
  wraps[p] = make_int4(W[0], W[1], W[2], 0);
}

struct NlWork {
  BinData b;
  int32_t *cnt;
  int64_t *off;
  TileList tl;  // large lists
  int4 *wraps;  // [N]
};

static void carve_nl(Carver &c, NlWork &w, int64_t n, int64_t ns) {
  carve_bins(c, w.b, n, ns);
  w.cnt = c.take<int32_t>(n);
  w.off = c.take<int64_t>(n + 1);
  carve_tiles(c, w.tl, n, ns);
  w.wraps = c.take<int4>(n);
}

// Up to these many atoms a list takes one warp per atom, beyond them one per tile: a tile
// is some 200 us of work for its warp in the two passes whatever the call, so few of them
// leave the GPU idle.  A whole call in us by warps and by tiles (full lists; half lists
// change over at the same size or some 15 % later), and by one thread per atom before both:
//   one system of argon    17,000 264, 335, 505   25,000 319, 351, 554   32,000 361, 331, 571
//                          45,000 437, 343, 639
//   copper, 8 to 512 each  17,000 274, 370, 522   32,000 377, 428, 573   45,000 463, 484, 622
//                          60,000 553, 453, 698
//   Kob-Andersen density,  18,000 541, 735, 1109  32,000 773, 740, 1371  45,000 997, 1052, 1821
//   64 to 1,000 each       60,000 1258, 1135, 2018
// Tiles of a large system are all full and alike; small systems cut theirs short and give
// windows of many short spans.  (256 atoms: 20 us for both passes, 276 us with one thread
// per atom.)
constexpr int64_t kNlWarpMaxAtoms = 49152;
constexpr int64_t kNlWarpMaxLarge = 28672;
constexpr int64_t kNlLargeSystem = 4096;  // mean size from which the second limit holds

template <class P>
static int nl_build(const P *pos, const P *cell, const uint8_t *pbc, const int64_t *sys,
                    int64_t n, int64_t ns, double cutoff, int flags, int64_t *mapping,
                    int64_t stride, int packed, int64_t *sysmap, P *shifts, int64_t cap,
                    int64_t *n_pairs, NlWork &w, cudaStream_t st) {
  // n bounds the largest system, so a small call takes the one-launch binning
  TSB_TRY(prepare_bins_any<P>(pos, cell, pbc, sys, n, ns, cutoff, w.b, st, nullptr, n));
  const NlOut<P> out{w.off, cap, packed, mapping, stride, sysmap, shifts};
  const bool small = n <= (n < kNlLargeSystem * ns ? kNlWarpMaxAtoms : kNlWarpMaxLarge);
  constexpr int threads = 32 * kWinWarps;
  const unsigned grid = grid_for(n, kWinWarps);
  auto tile_pass = [&](auto kernel) {
    kernel<<<tile_grid(kernel, 0), threads, 0, st>>>(w.b, n, w.tl, w.wraps, cutoff, flags, w.cnt,
                                                     out);
  };
  const bool half = flags & TSB_NL_HALF;
  if (small) {
    k_nl_warp<P, false><<<grid, threads, 0, st>>>(w.b, n, cutoff, flags, w.cnt, out);
  } else {
    TSB_TRY(window_tiles(w.b, n, ns, nullptr, 32, w.tl, st));
    k_nl_wraps<<<grid_for(n), kBlock, 0, st>>>(w.b.sidx, w.b.wrap, n, w.wraps);
    half ? tile_pass(k_nl_tile<P, false, true>) : tile_pass(k_nl_tile<P, false, false>);
  }
  TSB_TRY(exclusive_scan(w.cnt, w.off, n, w.b.scan_tmp, st));
  cudaMemcpyAsync(n_pairs, w.off + n, sizeof(int64_t), cudaMemcpyDeviceToDevice, st);
  if (cap > 0) {
    if (small)
      k_nl_warp<P, true><<<grid, threads, 0, st>>>(w.b, n, cutoff, flags, w.cnt, out);
    else {
      TSB_TRY(restart_tiles(w.tl, st));
      half ? tile_pass(k_nl_tile<P, true, true>) : tile_pass(k_nl_tile<P, true, false>);
    }
  }
  TSB_CHECK_LAUNCH();
  return TSB_OK;
}

}  // namespace tsb

using namespace tsb;

extern "C" size_t tsb_nl_workspace_size(int64_t n_atoms, int64_t n_systems) {
  Carver c(nullptr, (size_t)-1);
  NlWork w;
  carve_nl(c, w, n_atoms, n_systems);
  return c.off + 256;
}

static int nl_entry(const void *positions, const void *cell_row, const uint8_t *pbc,
                    const int64_t *system_idx, int64_t n_atoms, int64_t n_systems, int dtype,
                    double cutoff, int flags, int64_t *mapping, int64_t mapping_stride,
                    int packed, int64_t *system_mapping, void *shifts, int64_t capacity,
                    int64_t *n_pairs, void *workspace, size_t workspace_bytes, void *stream) {
  if (n_atoms < 0 || n_systems < 1 || !(cutoff > 0.0) || !n_pairs || !cell_row || !pbc)
    return TSB_ERR_INVALID_ARG;
  if (n_atoms > 0 && (!positions || !system_idx)) return TSB_ERR_INVALID_ARG;
  if (capacity > 0 && (!mapping || !system_mapping || !shifts || mapping_stride < capacity))
    return TSB_ERR_INVALID_ARG;
  if (dtype != TSB_F32 && dtype != TSB_F64) return TSB_ERR_INVALID_ARG;
  if (n_atoms >= (int64_t)1 << 30) return TSB_ERR_UNSUPPORTED;
  Carver c(workspace, workspace_bytes);
  NlWork w;
  carve_nl(c, w, n_atoms, n_systems);
  if (!c.ok || !workspace) return TSB_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_atoms == 0) {
    cudaMemsetAsync(n_pairs, 0, sizeof(int64_t), st);
    TSB_CHECK_LAUNCH();
    return TSB_OK;
  }
  if (dtype == TSB_F64)
    return nl_build<double>((const double *)positions, (const double *)cell_row, pbc,
                            system_idx, n_atoms, n_systems, cutoff, flags, mapping,
                            mapping_stride, packed, system_mapping, (double *)shifts, capacity,
                            n_pairs, w, st);
  return nl_build<float>((const float *)positions, (const float *)cell_row, pbc, system_idx,
                         n_atoms, n_systems, cutoff, flags, mapping, mapping_stride, packed,
                         system_mapping, (float *)shifts, capacity, n_pairs, w, st);
}

extern "C" int tsb_nl_build(const void *positions, const void *cell_row, const uint8_t *pbc,
                            const int64_t *system_idx, int64_t n_atoms, int64_t n_systems,
                            int dtype, double cutoff, int flags, int64_t *mapping,
                            int64_t mapping_stride, int64_t *system_mapping, void *shifts,
                            int64_t capacity, int64_t *n_pairs, void *workspace,
                            size_t workspace_bytes, void *stream) {
  return nl_entry(positions, cell_row, pbc, system_idx, n_atoms, n_systems, dtype, cutoff, flags,
                  mapping, mapping_stride, 0, system_mapping, shifts, capacity, n_pairs,
                  workspace, workspace_bytes, stream);
}

extern "C" int tsb_nl_build_packed(const void *positions, const void *cell_row,
                                   const uint8_t *pbc, const int64_t *system_idx,
                                   int64_t n_atoms, int64_t n_systems, int dtype, double cutoff,
                                   int flags, int64_t *mapping, int64_t *system_mapping,
                                   void *shifts, int64_t capacity, int64_t *n_pairs,
                                   void *workspace, size_t workspace_bytes, void *stream) {
  return nl_entry(positions, cell_row, pbc, system_idx, n_atoms, n_systems, dtype, cutoff, flags,
                  mapping, capacity, 1, system_mapping, shifts, capacity, n_pairs, workspace,
                  workspace_bytes, stream);
}
