// Fused neighbour search + pair energy/force/virial (drop-in for
// PairPotentialModel.forward, torch_sim/models/pair_potential.py:351-464).
//
// A warp works through the full neighbour set of an atom (candidates gathered by
// tsb_window.cuh), so forces need no atomics and the summation order is fixed
// (deterministic results).  Each unordered pair is evaluated from both ends; per-atom
// energies/virials take half of each visit, matching the half-list weights of
// pair_potential.py:402-441.
// Displacements are formed in FP64 from the wrapped FP64 positions; the pair
// function runs in R (float by default, double with TSB_MATH_FP64).
#include "tsb_pair.cuh"
#include "tsb_sysreduce.cuh"
#include "tsb_window.cuh"

namespace tsb {

// One pair's terms, added to a lane's sums: forces in R, energy and virial in FP64
// (R is FP32 by default; the per-system sums are FP64).
//
// ROUND: the FP32 force sums round each product and sum on its own, in the order of the
// search: a run of some hundred steps shows their last digits.  (2,048 ragged Morse
// systems, FP32: 688 us a call, 634 with fused steps in the order of the spans' spread.)
template <int POT, class R, bool VIR, bool ROUND>
struct PairSum {
  R fx, fy, fz;
  double ei, v[VIR ? 6 : 1];

  __device__ __forceinline__ void clear() {
    fx = fy = fz = 0;
    ei = 0.0;
#pragma unroll
    for (int k = 0; k < (VIR ? 6 : 1); ++k) v[k] = 0.0;
  }

  // adds the pair when `on` (a pair left out is evaluated all the same and its terms
  // replaced by zeros, so that the lanes of a warp stay together); returns fr
  template <bool FORCE = true>
  __device__ __forceinline__ R add(bool on, R rx, R ry, R rz, const PairPrm<R> &ij,
                                   const PairPrm<R> &ji) {
    const R r2 = rx * rx + ry * ry + rz * rz;
    R e, fr;  // fr = -(dV/dr)/r
    pair_eval<POT, R>(ij, r2, e, fr);
    // force-defined pairs: both directed pairs (i, j) and (j, i) of the reference's
    // full list act on i, so the force adds f_ij and f_ji and the virial takes half
    // of it (pair_potential.py:567-600, stress scale 1/2 for a full list)
    double vw = 1.0;
    if constexpr (POT == TSB_POT_PLIFE) {
      R e2, fr2;
      pair_eval<POT, R>(ji, r2, e2, fr2);
      fr += fr2;
      vw = 0.5;
    }
    fr = on ? fr : R(0);
    e = on ? e : R(0);
    const R gx = fr * rx, gy = fr * ry, gz = fr * rz;  // force on j
    if constexpr (FORCE && ROUND) {
      fx = __fsub_rn(fx, __fmul_rn(fr, rx));
      fy = __fsub_rn(fy, __fmul_rn(fr, ry));
      fz = __fsub_rn(fz, __fmul_rn(fr, rz));
    } else if constexpr (FORCE) {
      fx -= gx;
      fy -= gy;
      fz -= gz;
    }
    ei += (double)e;
    if constexpr (VIR) {
      v[0] += vw * (double)(rx * gx);
      v[1] += vw * (double)(ry * gy);
      v[2] += vw * (double)(rz * gz);
      v[3] += vw * (double)(ry * gz);
      v[4] += vw * (double)(rx * gz);
      v[5] += vw * (double)(rx * gy);
    }
    return fr;
  }
};

// results of atom i from its sums t[0..NA)
template <class P, bool VIR>
__device__ __forceinline__ void write_atom(int64_t i, const double *t, int flags, double vol,
                                           P *forces, P *energies, P *stresses, double *e_half,
                                           double *vir_half) {
  if (flags & TSB_OUT_FORCES)
    for (int c = 0; c < 3; ++c) forces[3 * i + c] = (P)t[c];
  // reference per-atom energies: each endpoint receives the full pair energy
  // (pair_potential.py:411-417 with weight 1 on both mapping rows)
  if (flags & TSB_OUT_ENERGIES) energies[i] = (P)t[3];
  e_half[i] = 0.5 * t[3];
  if constexpr (VIR) {
    for (int c = 0; c < 6; ++c) vir_half[6 * i + c] = 0.5 * t[4 + c];
    if (flags & TSB_OUT_STRESSES) {
      // per-atom stress: -1/2 sum_j r_ij (x) f_ij / V (pair_potential.py:262-272)
      const double c = -0.5 / vol;
      P *o = stresses + 9 * i;
      o[0] = (P)(c * t[4]); o[1] = (P)(c * t[9]); o[2] = (P)(c * t[8]);
      o[3] = (P)(c * t[9]); o[4] = (P)(c * t[5]); o[5] = (P)(c * t[7]);
      o[6] = (P)(c * t[8]); o[7] = (P)(c * t[7]); o[8] = (P)(c * t[6]);
    }
  }
}

// the pairs of one atom: displacement, species of the neighbour and, << 8, its offset in
// its span modulo 4
template <class R>
struct PairWin : WinSpans {
  static constexpr int kCap = 192;  // (more: several chunks)
  R x[kCap], y[kCap], z[kCap];
  uint16_t info[kCap];
};

template <class R, bool VIR>
struct PairWarpSmem {
  // FP32 pair math: the force sums decide the result's digits, so their order is kept:
  // four partial sums per component, each over every fourth candidate of a span in turn,
  // as four lanes per atom would take them
  static constexpr bool ORDERED = sizeof(R) == 4;
  static constexpr int NA = VIR ? 10 : 4;  // forces, energy, virial
  PairWin<R> win;
  // the force terms of 32 pairs, each product rounded on its own (rows eleven banks
  // apart, so that the lanes below read them side by side)
  float term[ORDERED ? 3 : 1][ORDERED ? 43 : 1];
  double acc[NA];
};

// Small calls: one warp per atom, every atom of the batch in flight at once.  Lanes
// are added in FP64 by exchange.  (LJ, 256 atoms, FP64: 10.1 us against 57.4 us with
// four lanes walking an atom's rows in turn.)
//
// Bound by latency (the gathering's loads, then shared memory), so by the warps in
// flight: only the pairs themselves are kept, as displacements (19 KB a block in FP32,
// 26 in FP64), and 7 (FP64: 6) blocks per SM are asked for, 72 (80) registers.  A whole
// call in us with everything kept and 5 blocks, with 7 (6), and with the four lanes per
// atom before both: FP32 pair arithmetic, 9,000 argon atoms 115, 110, 143; 20,000 161,
// 147, 156; 45,000 254, 222, 229; 60,000 312, 270, 270; 47,000 Kob-Andersen atoms 242,
// 201, 198.  FP64: 30,000 argon atoms 186, 175, 200; 47,000 Kob-Andersen atoms 222, 196,
// 189.  (5 blocks with the pairs alone: 238 and 222 at 45,000 and 47,000 in FP32.)
// Tried and dropped: a partial sum's terms packed side by side (273 us for 60,000).
template <int POT, class R, class P, bool VIR>
__global__ void __launch_bounds__(32 * kWinWarps, sizeof(R) == 4 ? 7 : 6)
    k_pair_warp(BinData b, int64_t n, const double *__restrict__ table, int nsp, double cutoff,
                int flags, P *forces, P *energies, P *stresses, double *e_half,
                double *vir_half, const uint8_t *__restrict__ sys_active) {
  using Warp = PairWarpSmem<R, VIR>;
  constexpr bool ORDERED = Warp::ORDERED;
  constexpr int NV = VIR ? 16 : 4;
  extern __shared__ __align__(16) char smem[];
  Warp *warps = (Warp *)smem;
  PairPrm<R> *prm = (PairPrm<R> *)(warps + kWinWarps);
  double *prc2 = (double *)(prm + nsp * nsp);
  for (int k = threadIdx.x; k < nsp * nsp; k += blockDim.x) {
    prm[k] = make_prm<R>(POT, table + 5 * k, cutoff);
    prc2[k] = pair_rc2(POT, table + 5 * k, cutoff);
  }
  __syncthreads();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  Warp &me = warps[threadIdx.x >> 5];
  const int64_t p = (int64_t)blockIdx.x * kWinWarps + (threadIdx.x >> 5);
  if (p >= n) return;
  const double4 w = b.spos[p];
  const int i = tag_atom(w.w);
  const int s = b.sys_of[i];
  if (sys_active && !sys_active[s]) return;
  const SysGeom &G = b.geom[s];
  const int si = min(max(tag_species(w.w), 0), nsp - 1);
  PairSum<POT, R, VIR, false> sum;
  sum.clear();
  float fo = 0.0f;  // ORDERED, lanes 0..11: component lane / 4, partial sum lane % 4
  PairWin<R> &S = me.win;
  auto inside = [&](const Cand &c) {  // FP64 decision
    const int sj = min(max(tag_species(c.w), 0), nsp - 1);
    return c.d2 < prc2[si * nsp + sj] && !(c.q == p && !(S.jx[c.k] | S.jy[c.k] | S.jz[c.k]));
  };
  auto put = [&](int at, const Cand &c) {
    S.x[at] = (R)c.dx;
    S.y[at] = (R)c.dy;
    S.z[at] = (R)c.dz;
    S.info[at] = (uint16_t)(min(max(tag_species(c.w), 0), nsp - 1) | ((c.q - S.q0[c.k]) & 3) << 8);
  };
  window_gather(S, G, b.spos, b.bin_start, w, inside, put, [&](int kept) {
    for (int t0 = 0; t0 < kept; t0 += 32) {
      const int t = t0 + lane;
      const bool on = t < kept;
      int share = 0;
      if (on) {
        const R rx = S.x[t], ry = S.y[t], rz = S.z[t];
        const int info = S.info[t], sj = info & 255;
        share = info >> 8;
        const R fr = sum.template add<!ORDERED>(true, rx, ry, rz, prm[si * nsp + sj],
                                                prm[sj * nsp + si]);
        if constexpr (ORDERED) {
          me.term[0][lane] = __fmul_rn(fr, rx);
          me.term[1][lane] = __fmul_rn(fr, ry);
          me.term[2][lane] = __fmul_rn(fr, rz);
        }
      }
      if constexpr (ORDERED) {
        // a partial sum's pairs: a mask of lanes, taken from the lowest up
        unsigned todo = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned m = __ballot_sync(full, on && share == k);
          if ((lane & 3) == k) todo = m;
        }
        __syncwarp();
        if (lane < 12) {
          const float *d = me.term[lane >> 2];
          while (todo) {
            const int k0 = __ffs(todo) - 1;
            todo &= todo - 1;
            const int k1 = todo ? __ffs(todo) - 1 : k0;  // (two reads in flight)
            const float d0 = d[k0], d1 = d[k1];
            fo = __fsub_rn(fo, d0);
            if (todo) fo = __fsub_rn(fo, d1);
            todo &= todo - 1;
          }
        }
        __syncwarp();
      }
    }
  });
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  v[0] = (double)sum.fx;
  v[1] = (double)sum.fy;
  v[2] = (double)sum.fz;
  v[3] = sum.ei;
  if constexpr (VIR)
    for (int k = 0; k < 6; ++k) v[4 + k] = sum.v[k];
  const double tot = warp_multi_sum<NV>(v);
  constexpr int W = 32 / NV;
  if (lane % W == 0 && lane / W < Warp::NA) me.acc[lane / W] = tot;
  if constexpr (ORDERED) {
    const int l = 4 * (lane % 3);
    const float a0 = __shfl_sync(full, fo, l), a1 = __shfl_sync(full, fo, l + 1);
    const float a2 = __shfl_sync(full, fo, l + 2), a3 = __shfl_sync(full, fo, l + 3);
    __syncwarp();
    if (lane < 3) me.acc[lane] = (double)((a0 + a2) + (a1 + a3));
  }
  __syncwarp();
  if (lane == 0)
    write_atom<P, VIR>(i, me.acc, flags, G.vol, forces, energies, stresses, e_half, vir_half);
}

// Large calls: one warp per tile, one lane per atom.  MONO: one species, whose row of
// the table stays in registers.
template <int POT, class R, class P, bool VIR, bool MONO>
__global__ void __launch_bounds__(32 * kWinWarps, sizeof(R) == 4 ? 6 : 4)
    k_pair_tile(BinData b, TileList tl, const double *__restrict__ table, int nsp,
                double cutoff, int flags, P *forces, P *energies, P *stresses, double *e_half,
                double *vir_half) {
  constexpr bool ROUND = sizeof(R) == 4;  // sums in search order
  extern __shared__ __align__(16) char smem[];
  TileSmem<false> *warps = (TileSmem<false> *)smem;
  PairPrm<R> *prm = (PairPrm<R> *)(warps + kWinWarps);
  double *prc2 = (double *)(prm + nsp * nsp);
  for (int k = threadIdx.x; k < nsp * nsp; k += blockDim.x) {
    prm[k] = make_prm<R>(POT, table + 5 * k, cutoff);
    prc2[k] = pair_rc2(POT, table + 5 * k, cutoff);
  }
  __syncthreads();
  const int wid = threadIdx.x >> 5;
  TileSmem<false> &S = warps[wid];
  const PairPrm<R> row0 = prm[0];
  const double rc2_0 = prc2[0];
  const int nt = *tl.n_tiles;
  TileQueue queue(tl);
  for (int g; (g = queue.take(tl, nt)) >= 0;) {
    const Tile T = tl.tiles[g];
    PairSum<POT, R, VIR, ROUND> sum;
    int si = 0;
    tile_gather<!ROUND>(
        S, b, T, tl.order, nullptr, cutoff,
        [&](const TileAtom &A) {
          sum.clear();
          si = min(max(tag_species(A.w.w), 0), nsp - 1);
        },
        [&](const TileAtom &A, int kept, float pre2) {
          for (int t0 = 0; t0 < kept;) {
            int nn, unused = 0;
            t0 = tile_scan<false>(S, A, t0, kept, pre2, nn, 0.0f, unused);
            const int most = __reduce_max_sync(0xffffffffu, nn);
            const uint8_t *note = S.note + (threadIdx.x & 31);
#pragma unroll sizeof(R) == 4 ? 2 : 1
            for (int k = 0; k < most; ++k) {
              bool on = k < nn;
              const int t = on ? note[k * kTileStride] : 0;
              const double dx = S.x[t] - A.w.x, dy = S.y[t] - A.w.y, dz = S.z[t] - A.w.z;
              const double d2 = dx * dx + dy * dy + dz * dz;
              const int sj = MONO ? 0 : min((int)S.spec[t], nsp - 1);
              on = on && d2 < (MONO ? rc2_0 : prc2[si * nsp + sj]) &&  // FP64 decision
                   !(d2 == 0.0 && S.j[t] == A.i);
              sum.add(on, (R)dx, (R)dy, (R)dz, MONO ? row0 : prm[si * nsp + sj],
                      MONO ? row0 : prm[sj * nsp + si]);
            }
            __syncwarp();
          }
        },
        [&](const TileAtom &A) {
          if (!A.have) return;
          double t[VIR ? 10 : 4] = {(double)sum.fx, (double)sum.fy, (double)sum.fz, sum.ei};
          if constexpr (VIR)
            for (int k = 0; k < 6; ++k) t[4 + k] = sum.v[k];
          write_atom<P, VIR>(tag_atom(A.w.w), t, flags, b.geom[T.sys].vol, forces, energies,
                             stresses, e_half, vir_half);
        });
  }
}

struct PairWork {
  BinData b;
  double *e_half;
  double *vir_half;
  double *part;  // [7 * ns * chunks] slice sums (chunks > 1 only)
  int chunks;
  TileList tl;  // large calls
};

static void carve_pair(Carver &c, PairWork &w, int64_t n, int64_t ns) {
  carve_bins(c, w.b, n, ns);
  w.e_half = c.take<double>(n);
  w.vir_half = c.take<double>(6 * n);
  w.chunks = reduce_chunks(n, ns);
  w.part = w.chunks > 1 ? c.take<double>(7 * ns * w.chunks) : nullptr;
  carve_tiles(c, w.tl, n, ns);
}

// Up to these many atoms a call takes one warp per atom, beyond them one per tile: a
// tile is some 190 us of work for its warp whatever the call, so few of them leave the
// GPU idle.  With FP32 pair math the limit is that of the four-lane order of the sums
// (k_pair_warp keeps the four-lane order, k_pair_tile the one-lane order that larger
// calls have).  In FP64, a call in us by warps and by tiles:
//   one system of argon   18,000 141, 164   30,000 175, 166   45,000 218, 188   60,000 262, 225
//   the same, soft sphere 18,000 139, 258   30,000 177, 265   45,000 224, 314   60,000 275, 396
//   copper, 8 to 512 each 18,000  92, 173   29,000 123, 190   46,000 173, 215   62,000 223, 268
//   Kob-Andersen mixtures 21,000 111, 202   31,000 146, 201   47,000 196, 221   67,000 261, 281
// The second limit is that of cheap pair functions in systems too large for their tiles
// to be cut short.
constexpr int64_t kPairWarpMaxAtoms = kGroupSearchMaxAtoms;
constexpr int64_t kPairWarpMaxLarge = 24576;
constexpr int64_t kPairLargeSystem = 4096;

template <int POT, class R, class P, bool VIR>
static int launch_forces(PairWork &w, int64_t n, int64_t ns, const double *table, int nsp,
                         double cutoff, int flags, P *forces, P *energies, P *stresses,
                         const uint8_t *active, cudaStream_t st) {
  using Warp = PairWarpSmem<R, VIR>;
  const size_t tab = (size_t)nsp * nsp * (sizeof(PairPrm<R>) + sizeof(double));
  auto room = [](auto kernel, size_t bytes) {
    if (bytes > 48 * 1024)
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    return bytes;
  };
  const bool small_systems = n < kPairLargeSystem * ns;
  const bool all = Warp::ORDERED || POT == TSB_POT_SOFT || small_systems;
  if (n <= (all ? kPairWarpMaxAtoms : kPairWarpMaxLarge)) {
    auto kernel = k_pair_warp<POT, R, P, VIR>;
    kernel<<<grid_for(n, kWinWarps), 32 * kWinWarps,
             room(kernel, kWinWarps * sizeof(Warp) + tab), st>>>(
        w.b, n, table, nsp, cutoff, flags, forces, energies, stresses, w.e_half, w.vir_half,
        active);
  } else {
    auto go = [&](auto kernel) {
      const size_t bytes = room(kernel, kWinWarps * sizeof(TileSmem<false>) + tab);
      const unsigned grid = tile_grid(kernel, bytes);
      // Batches of small systems take tiles of 16 atoms while those make at most two
      // rounds of the resident warps (FP32 113,664 atoms, FP64 75,776): half the work
      // for a warp where there are warps to spare.  Tiles of 16 and of 32, us: FP32,
      // copper of 70,000 atoms 259, 285, of 105,000 277, 305, of 131,000 313, 324, of
      // 197,000 412, 355; Kob-Andersen of 75,000 313, 305, of 85,000 320, 328, of 113,000
      // 338, 386, of 211,000 522, 432; FP64, Kob-Andersen of 67,000 239, 285, of 85,000
      // 281, 299, of 113,000 323, 318.  One large system: argon of 70,000 296, 272.
      const int width = small_systems && n <= (int64_t)32 * kWinWarps * grid ? 16 : 32;
      TSB_TRY(window_tiles(w.b, n, ns, active, width, w.tl, st));
      kernel<<<grid, 32 * kWinWarps, bytes, st>>>(w.b, w.tl, table, nsp, cutoff, flags, forces,
                                                  energies, stresses, w.e_half, w.vir_half);
      return TSB_OK;
    };
    if (nsp == 1)
      TSB_TRY(go(k_pair_tile<POT, R, P, VIR, true>));
    else
      TSB_TRY(go(k_pair_tile<POT, R, P, VIR, false>));
  }
  TSB_CHECK_LAUNCH();
  return TSB_OK;
}

template <class P>
static int pair_forward(int pot, const double *table, int nsp, const int32_t *species,
                        const P *pos, const P *cell, const uint8_t *pbc, const int64_t *sys,
                        int64_t n, int64_t ns, double cutoff, int flags, P *energy,
                        P *forces, P *stress, P *energies, P *stresses,
                        const uint8_t *active, int64_t max_sys, PairWork &w,
                        cudaStream_t st) {
  TSB_TRY(prepare_bins_any<P>(pos, cell, pbc, sys, n, ns, cutoff, w.b, st, species, max_sys));
  const bool f64 = flags & TSB_MATH_FP64;
  if (n > 0) {
    const bool vir = flags & (TSB_OUT_STRESS | TSB_OUT_STRESSES);
    auto go = [&](auto pot_c) {
      constexpr int POT = decltype(pot_c)::value;
      auto run = [&](auto launch) {
        return launch(w, n, ns, table, nsp, cutoff, flags, forces, energies, stresses, active,
                      st);
      };
      if (f64)
        return vir ? run(launch_forces<POT, double, P, true>)
                   : run(launch_forces<POT, double, P, false>);
      return vir ? run(launch_forces<POT, float, P, true>)
                 : run(launch_forces<POT, float, P, false>);
    };
    if (pot == TSB_POT_LJ)
      TSB_TRY(go(std::integral_constant<int, TSB_POT_LJ>()));
    else if (pot == TSB_POT_MORSE)
      TSB_TRY(go(std::integral_constant<int, TSB_POT_MORSE>()));
    else if (pot == TSB_POT_SOFT)
      TSB_TRY(go(std::integral_constant<int, TSB_POT_SOFT>()));
    else
      TSB_TRY(go(std::integral_constant<int, TSB_POT_PLIFE>()));
  }
  k_sys_reduce<P><<<dim3((unsigned)ns, (unsigned)w.chunks), kBlock, 0, st>>>(
      w.b.geom, w.e_half, w.vir_half, flags, energy, stress, active, w.chunks, w.part);
  if (w.chunks > 1)
    k_sys_final<P><<<grid_for(ns), kBlock, 0, st>>>(w.b.geom, w.part, ns, w.chunks, flags,
                                                     energy, stress, active);
  TSB_CHECK_LAUNCH();
  return TSB_OK;
}

}  // namespace tsb

using namespace tsb;

extern "C" size_t tsb_pair_workspace_size(int64_t n_atoms, int64_t n_systems) {
  Carver c(nullptr, (size_t)-1);
  PairWork w;
  carve_pair(c, w, n_atoms, n_systems);
  return c.off + 256;
}

extern "C" int tsb_pair_forward(int potential, const double *table, int n_species,
                                const int32_t *species, const void *positions,
                                const void *cell_row, const uint8_t *pbc,
                                const int64_t *system_idx, int64_t n_atoms,
                                int64_t n_systems, int dtype, double cutoff, int out_flags,
                                void *energy, void *forces, void *stress, void *energies,
                                void *stresses, const uint8_t *sys_active,
                                int64_t max_system_atoms, void *workspace,
                                size_t workspace_bytes, void *stream) {
  if (potential < TSB_POT_LJ || potential > TSB_POT_PLIFE) return TSB_ERR_INVALID_ARG;
  if (n_species < 1 || n_species > kMaxSpecies || !table) return TSB_ERR_INVALID_ARG;
  if (n_species > 1 && !species) return TSB_ERR_INVALID_ARG;
  if (n_atoms < 0 || n_systems < 1 || !(cutoff > 0.0) || !cell_row || !pbc || !energy)
    return TSB_ERR_INVALID_ARG;
  if (n_atoms > 0 && (!positions || !system_idx)) return TSB_ERR_INVALID_ARG;
  if ((out_flags & TSB_OUT_FORCES) && !forces) return TSB_ERR_INVALID_ARG;
  if ((out_flags & TSB_OUT_STRESS) && !stress) return TSB_ERR_INVALID_ARG;
  if ((out_flags & TSB_OUT_ENERGIES) && !energies) return TSB_ERR_INVALID_ARG;
  if ((out_flags & TSB_OUT_STRESSES) && !stresses) return TSB_ERR_INVALID_ARG;
  if (dtype != TSB_F32 && dtype != TSB_F64) return TSB_ERR_INVALID_ARG;
  if (n_atoms >= (int64_t)1 << 30) return TSB_ERR_UNSUPPORTED;
  Carver c(workspace, workspace_bytes);
  PairWork w;
  carve_pair(c, w, n_atoms, n_systems);
  if (!c.ok || !workspace) return TSB_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == TSB_F64)
    return pair_forward<double>(potential, table, n_species, species,
                                (const double *)positions, (const double *)cell_row, pbc,
                                system_idx, n_atoms, n_systems, cutoff, out_flags,
                                (double *)energy, (double *)forces, (double *)stress,
                                (double *)energies, (double *)stresses, sys_active,
                                max_system_atoms, w, st);
  return pair_forward<float>(potential, table, n_species, species, (const float *)positions,
                             (const float *)cell_row, pbc, system_idx, n_atoms, n_systems,
                             cutoff, out_flags, (float *)energy, (float *)forces,
                             (float *)stress, (float *)energies, (float *)stresses, sys_active,
                             max_system_atoms, w, st);
}
