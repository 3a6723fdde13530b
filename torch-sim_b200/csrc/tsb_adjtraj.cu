// Whole trajectories and adjoint sweeps of small systems, one block per system.
//
// tsb_adj_trajectory integrates velocity Verlet (torch_sim/integrators/nve.py:74-130)
// with species-matrix Lennard-Jones forces for many steps in one launch, and
// tsb_adj_sweep runs the discrete adjoint (tsb_adjoint.cu) back over the stored
// positions in one launch.  A system's positions, its Verlet list and the shift table
// stay in shared memory; a step is two block barriers.
//
// Why.  Step by step, a 200-step loss with gradients of 256 systems of 108 atoms took
// ~6,000 launches of 2-30 us (list checks, frames, forces, sums, kicks; 45 ms per loss
// and gradient, 15 ms of it in force and Hessian kernels).  Systems are independent,
// so nothing but the launches' ends synchronised them.  One block per system removes
// the launches; what remains is bound by the gathers of neighbour positions from
// shared memory (random 8-byte reads) and by FP64 issue.  The same loss and gradients:
// trajectory 2.3 ms, sweep 4.2 ms; with the histogram and its gradient (tsb_adjoint.cu,
// 0.28 and 0.13 ms) 7.3 ms in all against 45.4 ms.
//
// Lists.  Entry: neighbour | image code << 11, image S in {-1,0,1}^3 of the build's
// wrapped positions, within cutoff + skin; every thread of a block agrees to rebuild
// when an atom moved more than skin / 2 since the build (the barrier carries the
// vote).  Needs every periodic plane spacing >= cutoff + skin; a narrower cell, a
// full list or a system larger than the caller said is reported in `status` and the
// caller takes the general path.
#include "tsb_common.cuh"
#include "tsb_search.cuh"

namespace tsb {

constexpr int kBlkThreads = 512;
// The largest system: lists of ~160 neighbours fill a block's shared memory there.
// Against the general path (100 steps with gradients): 4 systems of 60 / 200 / 500 atoms
// 1.4 / 3.0 / 9.0 ms against 14.4 / 15.7 / 18.3, 256 of 200 / 500 4.8 / 17.5 against
// 24.5 / 36.9.
constexpr int kBlkMaxAtoms = 512;
constexpr int kBlkMaxSpecies = 4;

struct BlkSystem {
  const double *table;
  int nsp;
  const int32_t *species;
  const double *cell;
  const uint8_t *pbc;
  const int64_t *lo, *hi;
  double cutoff, skin;
  int cap, stride;      // list rows, and entries per row
  const double *inv_m;
  double dt;
  int32_t *status;
};

// Shared memory of a block (`vecs` more vectors per atom for the sweep: 2).  The
// leads' own values that change rarely sit here too, for registers' sake.
struct BlkSmem {
  double *x, *y, *z;     // positions in the build's frame
  double *rx, *ry, *rz;  // ... at the build
  double *wx, *wy, *wz;  // W C of each atom's wrap at the build
  double *vx, *vy, *vz;  // sweep: lam_p, the vector the Hessian acts on
  double *lx, *ly, *lz;  // sweep: lam_q
  double *C, *T;         // row cell, its inverse (u_k = sum_m x_m T[3 m + k]) [9] each
  double *sv;            // [27][3] S C
  float *svf;            // the same in FP32
  int32_t *per;          // [3] periodic axes, [1] the lists can hold the cell's pairs
  double *tab;           // per species pair: sigma^2, 4 eps or eps, ..., cutoff^2
  int32_t *cnt;
  uint16_t *list;
  uint8_t *spec;
};

__host__ __device__ inline size_t blk_bytes(int max_atoms, int stride, int cap, int nsp, int vecs) {
  return sizeof(double) * ((size_t)3 * max_atoms * (3 + vecs) + 18 + 81 + 5 * nsp * nsp) +
         sizeof(float) * 84 + sizeof(int32_t) * (4 + max_atoms) +
         sizeof(uint16_t) * (size_t)stride * cap +
         (size_t)((max_atoms + 15) / 16 * 16);
}

__device__ inline BlkSmem blk_carve(char *p, int max_atoms, int stride, int cap, int nsp,
                                    int vecs) {
  BlkSmem s;
  double *d = (double *)p;
  auto take = [&](size_t n) {
    double *r = d;
    d += n;
    return r;
  };
  s.x = take(max_atoms);
  s.y = take(max_atoms);
  s.z = take(max_atoms);
  s.rx = take(max_atoms);
  s.ry = take(max_atoms);
  s.rz = take(max_atoms);
  s.wx = take(max_atoms);
  s.wy = take(max_atoms);
  s.wz = take(max_atoms);
  s.vx = s.vy = s.vz = s.lx = s.ly = s.lz = nullptr;
  if (vecs) {
    s.vx = take(max_atoms);
    s.vy = take(max_atoms);
    s.vz = take(max_atoms);
    s.lx = take(max_atoms);
    s.ly = take(max_atoms);
    s.lz = take(max_atoms);
  }
  s.C = take(9);
  s.T = take(9);
  s.sv = take(81);
  s.tab = take(5 * nsp * nsp);
  s.svf = (float *)d;
  s.per = (int32_t *)(s.svf + 84);
  s.cnt = s.per + 4;
  s.list = (uint16_t *)(s.cnt + max_atoms);
  s.spec = (uint8_t *)(s.list + (size_t)stride * cap);
  return s;
}

// One thread's part of its system: LANES threads per atom, the first of them ("lead")
// holds the atom's state.
template <int LANES>
struct BlkThread {
  int n, a, lane;
  bool on;           // has an atom
  int64_t i;         // ... its index

  // whole block, barriers inside; false (for every thread) without lists.  A system of
  // more atoms than the block was sized for is reported before anything of it is touched.
  __device__ bool setup(const BlkSystem &B, BlkSmem &S, int64_t s, int max_atoms) {
    const int64_t lo = B.lo[s];
    if (B.hi[s] - lo > max_atoms) {
      if (threadIdx.x == 0) atomicMax(B.status, 1 << 30);
      return false;
    }
    n = (int)(B.hi[s] - lo);
    a = threadIdx.x / LANES;
    lane = threadIdx.x % LANES;
    on = a < n;
    i = lo + (on ? a : 0);
    if (on && lane == 0)
      S.spec[a] = (uint8_t)(B.species ? min(max(B.species[i], 0), B.nsp - 1) : 0);
    if (threadIdx.x == 0) {
      double *C = S.C, *T = S.T;
      for (int k = 0; k < 9; ++k) C[k] = B.cell[9 * s + k];
      const double d = C[0] * (C[4] * C[8] - C[5] * C[7]) - C[1] * (C[3] * C[8] - C[5] * C[6]) +
                       C[2] * (C[3] * C[7] - C[4] * C[6]);
      const bool frac = isfinite(d) && fabs(d) > 1e-12;
      const double id = frac ? 1.0 / d : 0.0;
      // the inverse of the row cell, row-major
      T[0] = (C[4] * C[8] - C[5] * C[7]) * id;
      T[1] = (C[2] * C[7] - C[1] * C[8]) * id;
      T[2] = (C[1] * C[5] - C[2] * C[4]) * id;
      T[3] = (C[5] * C[6] - C[3] * C[8]) * id;
      T[4] = (C[0] * C[8] - C[2] * C[6]) * id;
      T[5] = (C[2] * C[3] - C[0] * C[5]) * id;
      T[6] = (C[3] * C[7] - C[4] * C[6]) * id;
      T[7] = (C[1] * C[6] - C[0] * C[7]) * id;
      T[8] = (C[0] * C[4] - C[1] * C[3]) * id;
      int fits = 1;
      for (int k = 0; k < 3; ++k) {
        S.per[k] = frac && B.pbc[3 * s + k];
        // u_k = T[3 m + k] x_m: plane spacing 1 / |column k| against cutoff + skin
        const double t0 = T[k], t1 = T[3 + k], t2 = T[6 + k];
        if (S.per[k] && !(sqrt(t0 * t0 + t1 * t1 + t2 * t2) * (B.cutoff + B.skin) <= 1.0))
          fits = 0;
      }
      S.per[3] = fits && n > 0;
      if (!fits) atomicMax(B.status, 1 << 30);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 81; k += blockDim.x) {
      const int code = k / 3, m = k % 3;
      const int sx = code / 9 - 1, sy = (code / 3) % 3 - 1, sz = code % 3 - 1;
      S.sv[k] = sx * S.C[m] + sy * S.C[3 + m] + sz * S.C[6 + m];
      S.svf[k] = (float)S.sv[k];
    }
    return S.per[3];
  }

  // lead: the atom's position into the frame of the build
  __device__ __forceinline__ void place(BlkSmem &S, const double *q) const {
    S.x[a] = q[0] - S.wx[a];
    S.y[a] = q[1] - S.wy[a];
    S.z[a] = q[2] - S.wz[a];
  }

  // whole block, barriers inside: wrap the positions q (leads) and build the list
  __device__ void build(const BlkSystem &B, BlkSmem &S, const double *q) {
    if (on && lane == 0) {
      int W[3];
      for (int k = 0; k < 3; ++k) {
        const double u = S.T[k] * q[0] + S.T[3 + k] * q[1] + S.T[6 + k] * q[2];
        const double f = floor(u);
        W[k] = S.per[k] && isfinite(f) ? (int)fmin(fmax(f, -1e9), 1e9) : 0;
      }
      S.wx[a] = W[0] * S.C[0] + W[1] * S.C[3] + W[2] * S.C[6];
      S.wy[a] = W[0] * S.C[1] + W[1] * S.C[4] + W[2] * S.C[7];
      S.wz[a] = W[0] * S.C[2] + W[1] * S.C[5] + W[2] * S.C[8];
      place(S, q);
      S.rx[a] = S.x[a];
      S.ry[a] = S.y[a];
      S.rz[a] = S.z[a];
    }
    __syncthreads();
    const double rcs2 = (B.cutoff + B.skin) * (B.cutoff + B.skin);
    const unsigned gmask = (LANES == 32 ? 0xffffffffu : ((1u << LANES) - 1u))
                           << ((threadIdx.x & 31) / LANES * LANES);
    const unsigned below = gmask & ((1u << (threadIdx.x & 31)) - 1u);
    // FP32 first: coordinates below B0 = the cell's diagonal sum put the FP32 r^2
    // within 2^-20 B0^2 of the FP64 one
    double b0 = 0.0;
    for (int k = 0; k < 3; ++k)
      b0 += sqrt(S.C[3 * k] * S.C[3 * k] + S.C[3 * k + 1] * S.C[3 * k + 1] +
                 S.C[3 * k + 2] * S.C[3 * k + 2]);
    const bool open = !(S.per[0] && S.per[1] && S.per[2]);
    const float pre2 = open ? INFINITY : __double2float_ru(rcs2 + 4.0 * b0 * b0 * 0x1p-20);
    const double xi = on ? S.x[a] : 0.0, yi = on ? S.y[a] : 0.0, zi = on ? S.z[a] : 0.0;
    int c = 0;
    // (every lane of the warp takes the same number of turns)
    for (int j0 = 0; j0 < n; j0 += LANES) {
      const int j = j0 + lane;
      const bool has = on && j < n;
      const double dx = has ? S.x[j] - xi : 0.0, dy = has ? S.y[j] - yi : 0.0,
                   dz = has ? S.z[j] - zi : 0.0;
      const float fx = (float)dx, fy = (float)dy, fz = (float)dz;
      for (int code = 0; code < 27; ++code) {
        const float gx = fx + S.svf[3 * code], gy = fy + S.svf[3 * code + 1],
                    gz = fz + S.svf[3 * code + 2];
        bool hit = has && gx * gx + gy * gy + gz * gz < pre2;
        if (!__any_sync(0xffffffffu, hit)) continue;
        if (hit) {
          const int sx = code / 9 - 1, sy = (code / 3) % 3 - 1, sz = code % 3 - 1;
          const double ex = dx + S.sv[3 * code], ey = dy + S.sv[3 * code + 1],
                       ez = dz + S.sv[3 * code + 2];
          hit = ex * ex + ey * ey + ez * ez < rcs2 && (S.per[0] || !sx) &&
                (S.per[1] || !sy) && (S.per[2] || !sz) && !(code == 13 && j == a);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
          const int k = c + __popc(m & below);
          if (k < B.cap) S.list[(size_t)k * B.stride + a] = (uint16_t)(j | code << 11);
        }
        c += __popc(m & gmask);
      }
    }
    if (on && lane == 0) {
      S.cnt[a] = min(c, B.cap);
      if (c > B.cap) atomicMax(B.status, c);
    }
    __syncthreads();
  }

  // lead: has the atom moved too far for the list?
  __device__ __forceinline__ bool expired(const BlkSystem &B, const BlkSmem &S) const {
    const double dx = S.x[a] - S.rx[a], dy = S.y[a] - S.ry[a], dz = S.z[a] - S.rz[a];
    return dx * dx + dy * dy + dz * dz > 0.25 * B.skin * B.skin;
  }
};

// rows of the pair table in shared memory: sigma^2, eps, 1/sigma, 1/eps, cutoff^2
__device__ inline void blk_table(const BlkSystem &B, BlkSmem &S) {
  for (int k = threadIdx.x; k < B.nsp * B.nsp; k += blockDim.x) {
    const double sg = B.table[5 * k], ep = B.table[5 * k + 1];
    const double r = fmin(B.cutoff, B.table[5 * k + 3]);
    S.tab[5 * k] = sg * sg;
    S.tab[5 * k + 1] = ep;
    S.tab[5 * k + 2] = 1.0 / sg;
    S.tab[5 * k + 3] = 1.0 / ep;
    S.tab[5 * k + 4] = r * r;
  }
}

template <int LANES>
__device__ __forceinline__ double lanes_sum(double v) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// LJ force on the thread's atom (every lane of its group gets it)
template <int LANES>
__device__ __forceinline__ void blk_force(const BlkSystem &B, const BlkSmem &S,
                                          const BlkThread<LANES> &t, double *f) {
  double fx = 0.0, fy = 0.0, fz = 0.0;
  if (t.on) {
    const double xi = S.x[t.a], yi = S.y[t.a], zi = S.z[t.a];
    const double *row = S.tab + 5 * B.nsp * S.spec[t.a];
    const int c = S.cnt[t.a];
    for (int k = t.lane; k < c; k += LANES) {
      const int e = S.list[(size_t)k * B.stride + t.a], j = e & 2047;
      const double *sv = S.sv + 3 * (e >> 11);
      const double dx = S.x[j] - xi + sv[0], dy = S.y[j] - yi + sv[1], dz = S.z[j] - zi + sv[2];
      const double *q = row + 5 * S.spec[j];
      const double d2 = dx * dx + dy * dy + dz * dz;
      if (d2 < q[4] && d2 > 0.0) {
        const double ir2 = 1.0 / d2, s2 = q[0] * ir2, s6 = s2 * s2 * s2;
        const double fr = 24.0 * q[1] * (2.0 * s6 * s6 - s6) * ir2;  // -V'/r
        fx -= fr * dx;
        fy -= fr * dy;
        fz -= fr * dz;
      }
    }
  }
  f[0] = lanes_sum<LANES>(fx);
  f[1] = lanes_sum<LANES>(fy);
  f[2] = lanes_sum<LANES>(fz);
}

// `traj` (may be null): positions before each step; ckpt_q / ckpt_p (may be null):
// the state before every `every`-th step.
template <int LANES>
__global__ void __launch_bounds__(kBlkThreads, 2)
    k_adj_trajectory(BlkSystem B, int max_atoms, int64_t n_atoms, const double *q0,
                     const double *p0, int64_t n_steps, int64_t every, double *q_out,
                     double *p_out, double *ckpt_q, double *ckpt_p, double *traj) {
  extern __shared__ __align__(16) char smem[];
  BlkSmem S = blk_carve(smem, max_atoms, B.stride, B.cap, B.nsp, 0);
  BlkThread<LANES> t;
  blk_table(B, S);
  if (!t.setup(B, S, blockIdx.x, max_atoms)) {  // (the same for every thread)
    // the caller learns of it at the end: what it computes meanwhile reads real positions
    const int64_t end = 3 * B.hi[blockIdx.x];
    for (int64_t k = 3 * B.lo[blockIdx.x] + threadIdx.x; k < end; k += blockDim.x) {
      q_out[k] = q0[k];
      p_out[k] = p0[k];
    }
    return;
  }
  const bool lead = t.on && t.lane == 0;
  double q[3], p[3], f[3], im = 0.0;
  for (int m = 0; m < 3; ++m) {
    q[m] = q0[3 * t.i + m];
    p[m] = p0[3 * t.i + m];
  }
  im = B.inv_m[t.i];
  __syncthreads();
  t.build(B, S, q);
  blk_force<LANES>(B, S, t, f);
  const double half = B.dt / 2;
  for (int64_t k = 0; k < n_steps; ++k) {
    if (lead) {
      if (traj)
        for (int m = 0; m < 3; ++m) traj[3 * (k * n_atoms + t.i) + m] = q[m];
      if (ckpt_q && k % every == 0)
        for (int m = 0; m < 3; ++m) {
          ckpt_q[3 * (k / every * n_atoms + t.i) + m] = q[m];
          ckpt_p[3 * (k / every * n_atoms + t.i) + m] = p[m];
        }
      // each product and sum rounded on its own, as the tensor expressions of
      // nve.py:118-130 round them
      for (int m = 0; m < 3; ++m) {
        p[m] = __dadd_rn(p[m], __dmul_rn(f[m], half));
        q[m] = __dadd_rn(q[m], __dmul_rn(__dmul_rn(p[m], im), B.dt));
      }
    }
    __syncthreads();  // the last forces have read the positions
    bool far_ = false;
    if (lead) {
      t.place(S, q);
      far_ = t.expired(B, S);
    }
    if (__syncthreads_or(far_)) t.build(B, S, q);
    blk_force<LANES>(B, S, t, f);
    for (int m = 0; m < 3; ++m) p[m] = __dadd_rn(p[m], __dmul_rn(f[m], half));
  }
  if (lead)
    for (int m = 0; m < 3; ++m) {
      q_out[3 * t.i + m] = q[m];
      p_out[3 * t.i + m] = p[m];
    }
}

// The adjoint sweep over traj[n_steps - 1 .. 0]: lam_p += (dt/m) lam_q, lam_q -=
// c H lam_p, gradients += c dF/dtheta^T lam_p, c = dt (dt / 2 at step 0 when `first`).
// Pair terms as in tsb_ljhvp.cuh, in powers of 1/r^2 (no square root):
//   V'/r = -24 eps (2 s^12 - s^6) / r^2,  V'' - V'/r = 24 eps (28 s^12 - 8 s^6) / r^2
template <int LANES, int NS>
__global__ void __launch_bounds__(kBlkThreads, NS <= 2 ? 2 : 1)
    k_adj_sweep(BlkSystem B, int max_atoms, int64_t n_atoms, const double *traj,
                int64_t n_steps, int first, double *lam_q, double *lam_p, double *grad) {
  extern __shared__ __align__(16) char smem[];
  BlkSmem S = blk_carve(smem, max_atoms, B.stride, B.cap, B.nsp, 1);
  BlkThread<LANES> t;
  blk_table(B, S);
  if (!t.setup(B, S, blockIdx.x, max_atoms)) return;
  const bool lead = t.on && t.lane == 0;
  if (lead) {
    S.lx[t.a] = lam_q[3 * t.i];
    S.ly[t.a] = lam_q[3 * t.i + 1];
    S.lz[t.a] = lam_q[3 * t.i + 2];
    S.vx[t.a] = lam_p[3 * t.i];
    S.vy[t.a] = lam_p[3 * t.i + 1];
    S.vz[t.a] = lam_p[3 * t.i + 2];
    S.wx[t.a] = S.wy[t.a] = S.wz[t.a] = 0.0;
  }
  const double step_m = __dmul_rn(B.dt, B.inv_m[t.i]);
  double gs[NS], ge[NS];
#pragma unroll
  for (int u = 0; u < NS; ++u) gs[u] = ge[u] = 0.0;
  for (int64_t k = n_steps - 1; k >= 0; --k) {
    __syncthreads();  // the last step has read the positions and vectors
    double q[3] = {0.0, 0.0, 0.0};
    bool far_ = k == n_steps - 1;
    if (lead) {
      for (int m = 0; m < 3; ++m) q[m] = traj[3 * (k * n_atoms + t.i) + m];
      S.vx[t.a] = __dadd_rn(S.vx[t.a], __dmul_rn(S.lx[t.a], step_m));
      S.vy[t.a] = __dadd_rn(S.vy[t.a], __dmul_rn(S.ly[t.a], step_m));
      S.vz[t.a] = __dadd_rn(S.vz[t.a], __dmul_rn(S.lz[t.a], step_m));
      t.place(S, q);
      far_ = far_ || t.expired(B, S);
    }
    if (__syncthreads_or(far_)) t.build(B, S, q);
    const double coef = first && k == 0 ? B.dt / 2 : B.dt;
    double hx = 0.0, hy = 0.0, hz = 0.0;
    if (t.on) {
      const double xi = S.x[t.a], yi = S.y[t.a], zi = S.z[t.a];
      const double v0 = S.vx[t.a], v1 = S.vy[t.a], v2 = S.vz[t.a];
      const double *row = S.tab + 5 * B.nsp * S.spec[t.a];
      const int c = S.cnt[t.a];
      for (int e0 = t.lane; e0 < c; e0 += LANES) {
        const int e = S.list[(size_t)e0 * B.stride + t.a], j = e & 2047;
        const double *sv = S.sv + 3 * (e >> 11);
        const double dx = S.x[j] - xi + sv[0], dy = S.y[j] - yi + sv[1], dz = S.z[j] - zi + sv[2];
        const int sj = S.spec[j];
        const double *r = row + 5 * sj;
        const double d2 = dx * dx + dy * dy + dz * dz;
        if (!(d2 < r[4]) || !(d2 > 0.0)) continue;
        const double w0 = v0 - S.vx[j], w1 = v1 - S.vy[j], w2 = v2 - S.vz[j];
        const double ir2 = 1.0 / d2, s2 = r[0] * ir2, s6 = s2 * s2 * s2, s12 = s6 * s6;
        const double e24 = 24.0 * r[1] * ir2;
        const double vr = -e24 * (2.0 * s12 - s6);
        const double b = e24 * (28.0 * s12 - 8.0 * s6) * ir2 * (dx * w0 + dy * w1 + dz * w2);
        hx += b * dx + vr * w0;
        hy += b * dy + vr * w1;
        hz += b * dz + vr * w2;
        const double dv = coef * (dx * v0 + dy * v1 + dz * v2);
        const double de = vr * r[3] * dv;
        const double ds = -6.0 * e24 * r[2] * (4.0 * s12 - s6) * dv;
#pragma unroll
        for (int u = 0; u < NS; ++u)
          if (u == sj) {
            ge[u] += de;
            gs[u] += ds;
          }
      }
    }
    hx = lanes_sum<LANES>(hx);
    hy = lanes_sum<LANES>(hy);
    hz = lanes_sum<LANES>(hz);
    if (lead) {
      S.lx[t.a] -= coef * hx;
      S.ly[t.a] -= coef * hy;
      S.lz[t.a] -= coef * hz;
    }
  }
  if (lead) {
    lam_q[3 * t.i] = S.lx[t.a];
    lam_q[3 * t.i + 1] = S.ly[t.a];
    lam_q[3 * t.i + 2] = S.lz[t.a];
    lam_p[3 * t.i] = S.vx[t.a];
    lam_p[3 * t.i + 1] = S.vy[t.a];
    lam_p[3 * t.i + 2] = S.vz[t.a];
  }
  // parameter gradients: the lanes of an atom, then the atoms in order
#pragma unroll
  for (int u = 0; u < NS; ++u) {
    gs[u] = lanes_sum<LANES>(gs[u]);
    ge[u] = lanes_sum<LANES>(ge[u]);
    __syncthreads();
    if (lead) {
      S.x[t.a] = gs[u];
      S.y[t.a] = ge[u];
    }
    __syncthreads();
    if (u < B.nsp && (int)threadIdx.x < B.nsp) {
      const int si = threadIdx.x;
      double a = 0.0, b = 0.0;
      for (int j = 0; j < t.n; ++j)
        if (S.spec[j] == si) {
          a += S.x[j];
          b += S.y[j];
        }
      double *g = grad + ((size_t)blockIdx.x * B.nsp * B.nsp + si * B.nsp + u) * 2;
      g[0] += a;
      g[1] += b;
    }
  }
}

__global__ void k_blk_bounds(const int64_t *sys, int64_t n, int64_t *lo, int64_t *hi) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t s = sys[i];
  if (i == 0 || sys[i - 1] != s) lo[s] = i;
  if (i == n - 1 || sys[i + 1] != s) hi[s] = i + 1;
}

// the largest dynamic shared memory of a block
inline int blk_smem_limit() {
  int dev = 0, bytes = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return bytes;
}

static int blk_prepare(BlkSystem &B, const double *table, int nsp, const int32_t *species,
                       const double *cell, const uint8_t *pbc, const int64_t *system_idx,
                       int64_t n, int64_t ns, int64_t max_atoms, double cutoff, double skin,
                       int cap, const double *inv_m, double dt, int32_t *status, int vecs,
                       void *workspace, size_t workspace_bytes, cudaStream_t st) {
  if (nsp < 1 || nsp > kBlkMaxSpecies || !table || (nsp > 1 && !species) || n < 1 || ns < 1 ||
      !cell || !pbc || !system_idx || !inv_m || !status || !(cutoff > 0.0) || !(skin >= 0.0) ||
      cap < 1 || max_atoms < 1)
    return TSB_ERR_INVALID_ARG;
  if (max_atoms > kBlkMaxAtoms) return TSB_ERR_UNSUPPORTED;
  Carver c(workspace, workspace_bytes);
  int64_t *lo = c.take<int64_t>(2 * ns), *hi = lo ? lo + ns : nullptr;
  if (!c.ok || !workspace) return TSB_ERR_WORKSPACE;
  const int stride = (int)(max_atoms + 1) / 2 * 2;
  if (blk_bytes((int)max_atoms, stride, cap, nsp, vecs) > (size_t)blk_smem_limit())
    return TSB_ERR_CAPACITY;
  cudaMemsetAsync(lo, 0, 2 * sizeof(int64_t) * ns, st);  // and hi
  k_blk_bounds<<<grid_for(n), kBlock, 0, st>>>(system_idx, n, lo, hi);
  B = BlkSystem{table, nsp, species, cell, pbc, lo, hi, cutoff, skin, cap, stride, inv_m, dt,
                status};
  return TSB_OK;
}

// threads per atom: as many as the largest system leaves room for
template <class F>
static void blk_lanes(int64_t max_atoms, F &&go) {
  if (4 * max_atoms <= kBlkThreads)
    go(std::integral_constant<int, 4>());
  else if (2 * max_atoms <= kBlkThreads)
    go(std::integral_constant<int, 2>());
  else
    go(std::integral_constant<int, 1>());
}

template <class K>
static void blk_room(K kernel, size_t bytes) {
  if (bytes > 48 * 1024)
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace tsb

using namespace tsb;

extern "C" int tsb_adj_block_max_atoms(void) { return kBlkMaxAtoms; }

extern "C" int tsb_adj_block_max_neighbors(int64_t max_system_atoms, int n_species, int sweep) {
  if (max_system_atoms < 1 || max_system_atoms > kBlkMaxAtoms || n_species < 1 ||
      n_species > kBlkMaxSpecies)
    return 0;
  const int stride = (int)(max_system_atoms + 1) / 2 * 2;
  const int64_t room = (int64_t)blk_smem_limit() -
                       (int64_t)blk_bytes((int)max_system_atoms, stride, 0, n_species,
                                          sweep ? 2 : 0);
  return room > 0 ? (int)(room / (int64_t)(sizeof(uint16_t) * stride)) : 0;
}

extern "C" size_t tsb_adj_block_workspace_size(int64_t n_systems) {
  Carver c(nullptr, (size_t)-1);
  c.take<int64_t>(n_systems);
  c.take<int64_t>(n_systems);
  return c.off + 256;
}

extern "C" int tsb_adj_trajectory(const double *table, int n_species, const int32_t *species,
                                  const double *cell_row, const uint8_t *pbc,
                                  const int64_t *system_idx, int64_t n_atoms, int64_t n_systems,
                                  int64_t max_system_atoms, double cutoff, double skin,
                                  int max_neighbors, const double *inv_m, const double *q,
                                  const double *p, double dt, int64_t n_steps, int64_t every,
                                  double *q_out, double *p_out, double *ckpt_q, double *ckpt_p,
                                  double *traj, int32_t *status, void *workspace,
                                  size_t workspace_bytes, void *stream) {
  if (!q || !p || !q_out || !p_out || n_steps < 0 || every < 1 || (ckpt_q && !ckpt_p))
    return TSB_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  BlkSystem B;
  TSB_TRY(blk_prepare(B, table, n_species, species, cell_row, pbc, system_idx, n_atoms,
                      n_systems, max_system_atoms, cutoff, skin, max_neighbors, inv_m, dt,
                      status, 0, workspace, workspace_bytes, st));
  blk_lanes(max_system_atoms, [&](auto l) {
    constexpr int LANES = decltype(l)::value;
    auto kernel = k_adj_trajectory<LANES>;
    const size_t bytes = blk_bytes((int)max_system_atoms, B.stride, B.cap, n_species, 0);
    blk_room(kernel, bytes);
    const int threads = (int)(LANES * max_system_atoms + 31) / 32 * 32;
    kernel<<<(unsigned)n_systems, threads, bytes, st>>>(B, (int)max_system_atoms, n_atoms, q, p,
                                                        n_steps, every, q_out, p_out, ckpt_q,
                                                        ckpt_p, traj);
  });
  TSB_CHECK_LAUNCH();
  return TSB_OK;
}

extern "C" int tsb_adj_sweep(const double *table, int n_species, const int32_t *species,
                             const double *cell_row, const uint8_t *pbc,
                             const int64_t *system_idx, int64_t n_atoms, int64_t n_systems,
                             int64_t max_system_atoms, double cutoff, double skin,
                             int max_neighbors, const double *inv_m, const double *traj,
                             double dt, int64_t n_steps, int first, double *lam_q,
                             double *lam_p, double *grad_params, int32_t *status,
                             void *workspace, size_t workspace_bytes, void *stream) {
  if (!traj || !lam_q || !lam_p || !grad_params || n_steps < 0) return TSB_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  BlkSystem B;
  TSB_TRY(blk_prepare(B, table, n_species, species, cell_row, pbc, system_idx, n_atoms,
                      n_systems, max_system_atoms, cutoff, skin, max_neighbors, inv_m, dt,
                      status, 2, workspace, workspace_bytes, st));
  blk_lanes(max_system_atoms, [&](auto l) {
    constexpr int LANES = decltype(l)::value;
    auto go = [&](auto kernel) {
      const size_t bytes = blk_bytes((int)max_system_atoms, B.stride, B.cap, n_species, 2);
      blk_room(kernel, bytes);
      const int threads = (int)(LANES * max_system_atoms + 31) / 32 * 32;
      kernel<<<(unsigned)n_systems, threads, bytes, st>>>(B, (int)max_system_atoms, n_atoms,
                                                          traj, n_steps, first, lam_q, lam_p,
                                                          grad_params);
    };
    if (n_species == 1)
      go(k_adj_sweep<LANES, 1>);
    else if (n_species == 2)
      go(k_adj_sweep<LANES, 2>);
    else
      go(k_adj_sweep<LANES, 4>);
  });
  TSB_CHECK_LAUNCH();
  return TSB_OK;
}
