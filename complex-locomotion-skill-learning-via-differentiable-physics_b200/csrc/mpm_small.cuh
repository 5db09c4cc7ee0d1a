// mpm_small.cuh -- MLS-MPM rollouts of bodies whose grid fits in one CTA's shared
// memory: one CTA per env runs all substeps of the rollout (or of its reverse
// pass) in one launch.
//
// The general kernels (mpm_kernels.cuh) take two launches per substep and
// direction; a few hundred particles leave them launch-bound (2 envs of 400
// particles on a 32 x 32 grid: 8.7 us per particle launch, 6.5 us per grid
// launch).  Here the particle state and the grid stay in shared memory, and two
// block barriers separate the particle phase (G2P of f, P2G of f + 1) from the grid
// phase.  Scatters: a warp sums its runs of equal base cells (warp_runs), the run's
// first lane stores the stencil's sums in a table and links them into its base
// cell's list; the grid phase walks the lists of a node's 3^D base cells.  (Shared
// float atomics took 10.4 k of the forward substep's 17 k cycles, the lists take
// 3.6 k; red.global would cost two fences per substep.)  Runs beyond the table's
// size are added with atomics.  Every substep's state and grid are recorded, so
// the reverse pass recomputes nothing.  The arithmetic is Kern's, term by term.
//
// Measured on B200, 2 envs of 400 particles, 120 substeps, forward and reverse:
// 3.85 -> 1.60 ms (5.7 + 6.9 us per substep).  Bound by the instructions that one
// SM issues for an env: 13 warps of ~2.5 k per substep.
#pragma once
#include "mpm_kernels.cuh"
#include "mpm_small_host.h"

namespace cls {
namespace mpm {

// what a particle phase leaves for the grid phase: NV values per stencil node
template <typename R, int D, int NV>
struct Scatter {
  static constexpr int NN = Kern<R, D>::NN;
  R* table;    // [NN NV][cap] sums of a run of particles on one base cell
  int* next;   // [cap] next run of the base cell
  int* head;   // [2][nodes] first run of a base cell, -1: none; of this phase and the next
  R* over;     // [NV][nodes] sums of the runs beyond cap
  int* count;  // [2] runs of this phase and the next
  int* slab;   // [2][2] their base cells' range along the first axis (min, max)
  int* node;   // [nodes] coordinates (10 bits each), bit 30: wall
};

constexpr int kSmallAhead = 3;   // grid nodes per thread loaded ahead in the reverse pass

struct SmallCarver {
  char* base;
  size_t off;
  template <typename T>
  __host__ __device__ T* take(size_t n) {
    T* p = reinterpret_cast<T*>(base + off);
    off += (sizeof(T) * n + 31) & ~size_t(31);
    return p;
  }
  template <typename R, int D, int NV>
  __host__ __device__ Scatter<R, D, NV> scatter(int nodes, int cap) {
    Scatter<R, D, NV> z;
    z.table = take<R>((size_t)z.NN * NV * cap);
    z.next = take<int>(cap);
    z.head = take<int>(2 * (size_t)nodes);
    z.over = take<R>((size_t)NV * nodes);
    z.count = take<int>(2);
    z.slab = take<int>(4);
    z.node = take<int>(nodes);
    return z;
  }
};

template <typename R, int D>
struct SmallFwdShared {
  R* x;        // [D][P]
  R* F;        // [D D][P]
  V4<R>* gv;   // [nodes] velocity, mass
  Scatter<R, D, D + 1> sc;  // momentum, mass
};
template <typename R, int D>
struct SmallAdjShared {
  R* ax;       // [D][P]
  R* aF;       // [D D][P]
  V4<R>* ga;   // [nodes] d (velocity before the update), d mass
  V4<R>* gv;   // [nodes] grid of the step at hand
  Scatter<R, D, D> sc;      // d velocity
};
template <typename R, int D>
__host__ __device__ inline size_t carve(char* base, int P, int nodes, int cap, SmallFwdShared<R, D>* s) {
  SmallCarver m{base, 0};
  SmallFwdShared<R, D> z;
  z.gv = m.take<V4<R>>(nodes);
  z.x = m.take<R>((size_t)D * P);
  z.F = m.take<R>((size_t)D * D * P);
  z.sc = m.scatter<R, D, D + 1>(nodes, cap);
  if (s) *s = z;
  return m.off;
}
template <typename R, int D>
__host__ __device__ inline size_t carve(char* base, int P, int nodes, int cap, SmallAdjShared<R, D>* s) {
  SmallCarver m{base, 0};
  SmallAdjShared<R, D> z;
  z.ga = m.take<V4<R>>(nodes);
  z.gv = m.take<V4<R>>(nodes);
  z.ax = m.take<R>((size_t)D * P);
  z.aF = m.take<R>((size_t)D * D * P);
  z.sc = m.scatter<R, D, D>(nodes, cap);
  if (s) *s = z;
  return m.off;
}

// dense node index inside an env's grid
template <int D>
__device__ __forceinline__ int small_node(int n_grid, const int I[D]) {
  int n = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) n = n * n_grid + I[d];
  return n;
}

// no runs in buffer `buf` (one thread)
template <typename R, int D, int NV>
__device__ __forceinline__ void scatter_clear(const Scatter<R, D, NV>& sc, int buf) {
  sc.count[buf] = 0;
  sc.slab[2 * buf] = INT_MAX;
  sc.slab[2 * buf + 1] = INT_MIN;
}

// empty lists and overflow sums, node coordinates and walls; the caller
// synchronises
template <typename R, int D, int NV>
__device__ __forceinline__ void scatter_init(const Scatter<R, D, NV>& sc, int nodes, int n_grid, int bound) {
  for (int i = threadIdx.x; i < nodes; i += blockDim.x) {
    sc.head[i] = sc.head[nodes + i] = -1;
#pragma unroll
    for (int k = 0; k < NV; ++k) sc.over[k * nodes + i] = 0;
    int r = i, pk = 0;
    bool wall = false;
#pragma unroll
    for (int d = D - 1; d >= 0; --d) {
      const int c = r % n_grid;
      r /= n_grid;
      pk |= c << (10 * d);
      wall |= (c < bound || c > n_grid - bound);
    }
    sc.node[i] = pk | (wall ? 1 << 30 : 0);
  }
  if (threadIdx.x < 2) scatter_clear<R, D, NV>(sc, threadIdx.x);
}

// where a run's sums go (its first lane): the table slot, linked into the base
// cell's list of buffer `buf`, or beyond the table
template <typename R, int D, int NV>
__device__ __forceinline__ int scatter_slot(const Scatter<R, D, NV>& sc, const WarpRuns& runs, bool valid, int nodes,
                                            int cap, int buf, int cell, int base0) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int lo = __reduce_min_sync(full, valid ? base0 : INT_MAX), hi = __reduce_max_sync(full, valid ? base0 : INT_MIN);
  if (lane == 0 && lo <= hi) {
    atomicMin(sc.slab + 2 * buf, lo);
    atomicMax(sc.slab + 2 * buf + 1, hi);
  }
  const unsigned heads = __ballot_sync(full, valid && runs.head);
  int first = 0;
  if (lane == 0 && heads) first = atomicAdd(sc.count + buf, __popc(heads));
  first = __shfl_sync(full, first, 0);
  const int slot = first + __popc(heads & ((1u << lane) - 1));
  if (valid && runs.head && slot < cap) sc.next[slot] = atomicExch(sc.head + buf * nodes + cell, slot);
  return slot;
}

// v summed over each run; its first lane stores or adds them for stencil node nq
template <typename R, int D, int NV>
__device__ __forceinline__ void scatter_add(const Scatter<R, D, NV>& sc, const WarpRuns& runs, bool valid, int nodes,
                                            int cap, int slot, int nq, int node, R (&v)[NV]) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  for (int s = 0, off = 1; s < runs.steps; ++s, off <<= 1) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      const R o = __shfl_down_sync(full, v[k], off);
      if (lane + off <= runs.last) v[k] += o;
    }
  }
  if (valid && runs.head) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (slot < cap) sc.table[(nq * NV + k) * cap + slot] = v[k];
      else atomicAdd(sc.over + k * nodes + node, v[k]);
    }
  }
}

// the sums of node i, from the lists of buffer `buf` (and what lies beyond the
// table, which it empties)
template <typename R, int D, int NV>
__device__ __forceinline__ void scatter_take(const Scatter<R, D, NV>& sc, int nodes, int cap, int buf, int n_grid, int i,
                                             bool over, R (&v)[NV]) {
  const int pk = sc.node[i];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    v[k] = 0;
    if (over) {
      v[k] = sc.over[k * nodes + i];
      sc.over[k * nodes + i] = 0;
    }
  }
  int run[Scatter<R, D, NV>::NN];
#pragma unroll
  for (int nq = 0; nq < Scatter<R, D, NV>::NN; ++nq) {
    int o[D], off = 0;
    Kern<R, D>::offs(nq, o);
    bool ok = true;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const int b = ((pk >> (10 * d)) & 1023) - o[d];
      ok = ok && b >= 0 && b <= n_grid - 3;
      off = off * n_grid + o[d];
    }
    run[nq] = ok ? sc.head[buf * nodes + i - off] : -1;
  }
#pragma unroll
  for (int nq = 0; nq < Scatter<R, D, NV>::NN; ++nq) {
    for (int r = run[nq]; r >= 0; r = sc.next[r]) {
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] += sc.table[(nq * NV + k) * cap + r];
    }
  }
}

// the other buffer's lists emptied for the next phase; the nodes that buffer
// `buf`'s runs reach: whole slabs [x, y) along the first axis (a quarter to a half
// of the grid; every body has at least one run)
template <typename R, int D, int NV>
__device__ __forceinline__ int2 scatter_turn(const Scatter<R, D, NV>& sc, int nodes, int n_grid, int buf) {
  for (int i = threadIdx.x; i < nodes; i += blockDim.x) sc.head[(buf ^ 1) * nodes + i] = -1;
  if (threadIdx.x == 0) scatter_clear<R, D, NV>(sc, buf ^ 1);
  const int row = nodes / n_grid;
  return make_int2(sc.slab[2 * buf] * row, (sc.slab[2 * buf + 1] + 3) * row);
}

// Rollout of a.steps substeps: records[t] holds x, v, C, F and the grid of step t
// (t = 0: the state it starts from), fin the state after the last.
template <typename R, int D>
__global__ void __launch_bounds__(kSmallThreads) mpm_small_fwd_kernel(SmallFwdArgs<R> a) {
  using K = Kern<R, D>;
  extern __shared__ __align__(32) char small_smem[];
  const Phys<R>& c = a.c;
  const int P = c.P, n = c.n_grid, tid = threadIdx.x, nt = blockDim.x, e = blockIdx.x;
  int nodes = 1;
#pragma unroll
  for (int d = 0; d < D; ++d) nodes *= n;
  SmallFwdShared<R, D> s;
  carve<R, D>(small_smem, P, nodes, a.cap, &s);
  const long long EP = c.EP, q0 = (long long)e * P;
  for (int p = tid; p < P; p += nt) {
#pragma unroll
    for (int d = 0; d < D; ++d) s.x[d * P + p] = a.x0[d * EP + q0 + p];
#pragma unroll
    for (int i = 0; i < D * D; ++i) s.F[i * P + p] = a.F0[i * EP + q0 + p];
  }
  scatter_init<R, D, D + 1>(s.sc, nodes, n, c.bound);
  const size_t slab = (size_t)c.E * c.nblk * Blk<D>::NODES, goff = (size_t)e * c.nblk * Blk<D>::NODES;
  __syncthreads();
  for (int f = 0; f <= a.steps; ++f) {
    // ---- particles: G2P of step f - 1, then P2G of step f
    for (int p0 = 0; p0 < P; p0 += nt) {
      const int p = p0 + tid;
      const bool valid = p < P;
      R x[D], v[D], Cm[D * D];
      int base[D];
      R fx[D], w[3][D], dw[3][D];
#pragma unroll
      for (int d = 0; d < D; ++d) x[d] = valid ? s.x[d * P + p] : R(0);
      if (f > 0) {
        K::weights(x, c.inv_dx, n, base, fx, w, dw);
#pragma unroll
        for (int i = 0; i < D; ++i) v[i] = 0;
#pragma unroll
        for (int i = 0; i < D * D; ++i) Cm[i] = 0;
#pragma unroll
        for (int nq = 0; nq < K::NN; ++nq) {
          int o[D], I[D];
          K::offs(nq, o);
          const R wt = K::wgt(w, o);
#pragma unroll
          for (int d = 0; d < D; ++d) I[d] = base[d] + o[d];
          const V4<R> g4 = s.gv[small_node<D>(n, I)];
          const R g[3] = {g4.x, g4.y, g4.z};
          const R s4 = R(4) * wt * c.inv_dx;
#pragma unroll
          for (int i = 0; i < D; ++i) {
            v[i] += wt * g[i];
#pragma unroll
            for (int j = 0; j < D; ++j) Cm[i * D + j] += s4 * g[i] * ((R)o[j] - fx[j]);
          }
        }
        const bool last = f == a.steps;
        R* xo = last ? a.fin_x : a.rec_x + (size_t)f * EP * D;
        R* vo = last ? a.fin_v : a.rec_v + (size_t)f * EP * D;
        R* Co = last ? a.fin_C : a.rec_C + (size_t)f * EP * D * D;
        if (valid) {
#pragma unroll
          for (int i = 0; i < D; ++i) {
            x[i] += c.dt * v[i];
            s.x[i * P + p] = x[i];
            xo[i * EP + q0 + p] = x[i];
            vo[i * EP + q0 + p] = v[i];
          }
#pragma unroll
          for (int i = 0; i < D * D; ++i) Co[i * EP + q0 + p] = Cm[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < D; ++i) v[i] = valid ? a.v0[i * EP + q0 + p] : R(0);
#pragma unroll
        for (int i = 0; i < D * D; ++i) Cm[i] = valid ? a.C0[i * EP + q0 + p] : R(0);
      }
      {
        R sum[D];
        const R pwv = valid ? ld(c.pw + p) : R(0);
#pragma unroll
        for (int d = 0; d < D; ++d) sum[d] = pwv * x[d];
        warp_sum_add<R, D>(sum, a.csum + ((size_t)f * c.E + e) * D);
      }
      if (f == a.steps) continue;
      K::weights(x, c.inv_dx, n, base, fx, w, dw);
      R aff[D * D];
      {
        R F[D * D], nF[D * D], tau[D * D], fb[D], am = 0;
#pragma unroll
        for (int i = 0; i < D * D; ++i) F[i] = valid ? s.F[i * P + p] : R(i % (D + 1) == 0);
        K::new_F(Cm, F, c.dt, nF);
        const int m = valid ? ld(c.muscle + p) : -1;
#pragma unroll
        for (int d = 0; d < D; ++d) fb[d] = 0;
        if (m >= 0) {
          am = ld(a.act + ((size_t)f * c.E + e) * c.M + m) * c.act_strength;
#pragma unroll
          for (int d = 0; d < D; ++d) fb[d] = ld(c.fibre + (long long)d * P + p);
        }
        K::stress(c, nF, m >= 0, am, fb, tau);
#pragma unroll
        for (int i = 0; i < D * D; ++i) aff[i] = (-c.ks * tau[i] + c.mass * Cm[i]) * c.dx;
        if (valid) {
          R* Fo = f + 1 == a.steps ? a.fin_F : a.rec_F + (size_t)(f + 1) * EP * D * D;
#pragma unroll
          for (int i = 0; i < D * D; ++i) {
            s.F[i * P + p] = nF[i];
            Fo[i * EP + q0 + p] = nF[i];
          }
        }
      }
      const WarpRuns runs = warp_runs<D>(valid, base);
      const int slot = scatter_slot<R, D, D + 1>(s.sc, runs, valid, nodes, a.cap, f & 1, small_node<D>(n, base), base[0]);
#pragma unroll 1
      for (int ol = 0; ol < (D == 3 ? 3 : 1); ++ol) {
        const R wl = D == 3 ? (ol == 0 ? w[0][D - 1] : (ol == 1 ? w[1][D - 1] : w[2][D - 1])) : R(1);
#pragma unroll
        for (int nq = 0; nq < 9; ++nq) {
          int o[D], I[D];
          o[0] = nq % 3;
          o[1] = nq / 3;
          if (D == 3) o[D - 1] = ol;
          const R wt = w[o[0]][0] * w[o[1]][1] * wl;
          R val[D + 1];
#pragma unroll
          for (int i = 0; i < D; ++i) {
            R m = c.mass * v[i];
#pragma unroll
            for (int j = 0; j < D; ++j) m += aff[i * D + j] * ((R)o[j] - fx[j]);
            val[i] = valid ? wt * m : R(0);
            I[i] = base[i] + o[i];
          }
          val[D] = valid ? wt * c.mass : R(0);
          scatter_add<R, D, D + 1>(s.sc, runs, valid, nodes, a.cap, slot, nq + 9 * ol, small_node<D>(n, I), val);
        }
      }
    }
    if (f == a.steps) break;
    __syncthreads();
    // ---- grid update of step f
    V4<R>* go = a.grid + (size_t)f * slab + goff;
    const bool over = s.sc.count[f & 1] > a.cap;
    const int2 span = scatter_turn<R, D, D + 1>(s.sc, nodes, n, f & 1);
    for (int i = span.x + tid; i < span.y; i += nt) {
      R m[D + 1];
      scatter_take<R, D, D + 1>(s.sc, nodes, a.cap, f & 1, n, i, over, m);
      const R inv_m = rcp_s<R>(m[D] + R(1e-10));
      V4<R> o;
      o.x = inv_m * m[0];
      o.y = inv_m * m[1] + c.dt * c.gravity;
      o.z = D == 3 ? inv_m * m[D - 1] : R(0);
      if (s.sc.node[i] >> 30) o.x = o.y = o.z = 0;
      o.w = m[D];
      s.gv[i] = o;
      go[i] = o;
    }
    __syncthreads();
  }
}

// Reverse pass over the recorded rollout.
template <typename R, int D>
__global__ void __launch_bounds__(kSmallThreads) mpm_small_adj_kernel(SmallAdjArgs<R> a) {
  using K = Kern<R, D>;
  extern __shared__ __align__(32) char small_smem[];
  const Phys<R>& c = a.c;
  const int P = c.P, n = c.n_grid, tid = threadIdx.x, nt = blockDim.x, e = blockIdx.x, lane = tid & 31;
  int nodes = 1;
#pragma unroll
  for (int d = 0; d < D; ++d) nodes *= n;
  SmallAdjShared<R, D> s;
  carve<R, D>(small_smem, P, nodes, a.cap, &s);
  const long long EP = c.EP, q0 = (long long)e * P;
  const size_t slab = (size_t)c.E * c.nblk * Blk<D>::NODES, goff = (size_t)e * c.nblk * Blk<D>::NODES;
  for (int i = tid; i < nodes; i += nt) {
    s.gv[i] = a.grid[(size_t)(a.steps - 1) * slab + goff + i];
  }
  scatter_init<R, D, D>(s.sc, nodes, n, c.bound);
  __syncthreads();
  // f = steps: the loss seed and G2P^T of the last step; then P2G^T of f, seed of
  // f and G2P^T of f - 1
  for (int f = a.steps; f >= 0; --f) {
    const R* rx = f > 0 ? a.rec_x + (size_t)f * EP * D : a.x0;
    const R* rv = f > 0 ? a.rec_v + (size_t)f * EP * D : a.v0;
    const R* rC = f > 0 ? a.rec_C + (size_t)f * EP * D * D : a.C0;
    const R* rF = f > 0 ? a.rec_F + (size_t)f * EP * D * D : a.F0;
    const R* rh = f > 1 ? a.rec_x + (size_t)(f - 1) * EP * D : a.x0;
    const R seed_w = a.seed_w[f];
    if (f < a.steps) {
      // ---- grid adjoint of step f; the grid of step f - 1 takes its place
      const bool over = s.sc.count[(f + 1) & 1] > a.cap;
      const int2 span = scatter_turn<R, D, D>(s.sc, nodes, n, (f + 1) & 1);
      // the grid of the step before, loaded ahead of the lists' walk
      V4<R> before[kSmallAhead];
#pragma unroll
      for (int k = 0; k < kSmallAhead; ++k)
        if (f > 0 && tid + k * nt < nodes) before[k] = a.grid[(size_t)(f - 1) * slab + goff + tid + k * nt];
      for (int i = span.x + tid; i < span.y; i += nt) {
        R v[D];
        scatter_take<R, D, D>(s.sc, nodes, a.cap, (f + 1) & 1, n, i, over, v);
        const R g[3] = {v[0], v[1], D == 3 ? v[D - 1] : R(0)};
        const V4<R> sv = s.gv[i];
        const R inv_m = rcp_s<R>(sv.w + R(1e-10));
        V4<R> o{0, 0, 0, 0};
        if (!(s.sc.node[i] >> 30)) {
          const R vy = sv.y - c.dt * c.gravity;
          o.x = g[0] * inv_m;
          o.y = g[1] * inv_m;
          o.z = D == 3 ? g[2] * inv_m : R(0);
          o.w = -(g[0] * sv.x + g[1] * vy + (D == 3 ? g[2] * sv.z : R(0))) * inv_m;
        }
        s.ga[i] = o;
      }
      __syncthreads();  // the grid of step f is read
#pragma unroll
      for (int k = 0; k < kSmallAhead; ++k)
        if (f > 0 && tid + k * nt < nodes) s.gv[tid + k * nt] = before[k];
      if (f > 0)
        for (int i = tid + kSmallAhead * nt; i < nodes; i += nt) s.gv[i] = a.grid[(size_t)(f - 1) * slab + goff + i];
      __syncthreads();
    }
    for (int p0 = 0; p0 < P; p0 += nt) {
      const int p = p0 + tid;
      const bool valid = p < P;
      const long long q = q0 + (valid ? p : 0);
      int base[D];
      R fx[D], w[3][D], dw[3][D], ax[D], av[D], aC[D * D], aFo[D * D];
      R seed[D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        seed[d] = 0;
        if (seed_w != R(0) && valid)
          seed[d] = R(2) * seed_w * center_error<R>(a.csum[((size_t)f * c.E + e) * D + d], a.pw_sum,
                                                    ld(a.target + ((size_t)f * c.E + e) * D + d)) *
                    ld(c.pw + p) / a.pw_sum;
      }
      if (f < a.steps) {
        R x[D], vp[D], Cp[D * D], Fp[D * D], nF[D * D], aff[D * D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          x[d] = ld(rx + d * EP + q);
          vp[d] = ld(rv + d * EP + q);
        }
#pragma unroll
        for (int i = 0; i < D * D; ++i) {
          Cp[i] = ld(rC + i * EP + q);
          Fp[i] = ld(rF + i * EP + q);
        }
        K::weights(x, c.inv_dx, n, base, fx, w, dw);
        const int m = valid ? ld(c.muscle + p) : -1;
        R fb[D], am = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) fb[d] = 0;
        if (m >= 0) {
          am = ld(a.act + ((size_t)f * c.E + e) * c.M + m) * c.act_strength;
#pragma unroll
          for (int d = 0; d < D; ++d) fb[d] = ld(c.fibre + (long long)d * P + p);
        }
        K::new_F(Cp, Fp, c.dt, nF);
        {
          R tau[D * D];
          K::stress(c, nF, m >= 0, am, fb, tau);
#pragma unroll
          for (int i = 0; i < D * D; ++i) aff[i] = (-c.ks * tau[i] + c.mass * Cp[i]) * c.dx;
        }
        R gaff[D * D], gfx[D];
#pragma unroll
        for (int i = 0; i < D * D; ++i) gaff[i] = 0;
#pragma unroll
        for (int i = 0; i < D; ++i) gfx[i] = av[i] = 0;
#pragma unroll
        for (int nq = 0; nq < K::NN; ++nq) {
          int o[D], I[D];
          K::offs(nq, o);
          const R wt = K::wgt(w, o);
          R dwt[D], dp[D];
          K::dwgt(w, dw, o, dwt);
#pragma unroll
          for (int d = 0; d < D; ++d) {
            dp[d] = (R)o[d] - fx[d];
            I[d] = base[d] + o[d];
          }
          const V4<R> g4 = s.ga[small_node<D>(n, I)];
          const R gg[3] = {g4.x, g4.y, g4.z};
          R gw = g4.w * c.mass;
#pragma unroll
          for (int i = 0; i < D; ++i) {
            R mom = c.mass * vp[i];
#pragma unroll
            for (int j = 0; j < D; ++j) mom += aff[i * D + j] * dp[j];
            gw += gg[i] * mom;
            av[i] += wt * c.mass * gg[i];
            const R wg = wt * gg[i];
#pragma unroll
            for (int j = 0; j < D; ++j) gaff[i * D + j] += wg * dp[j];
          }
#pragma unroll
          for (int j = 0; j < D; ++j) {
            R acc = 0;
#pragma unroll
            for (int i = 0; i < D; ++i) acc += aff[i * D + j] * gg[i];
            gfx[j] -= wt * acc;
          }
#pragma unroll
          for (int d = 0; d < D; ++d) gfx[d] += gw * dwt[d];
        }
        R gnF[D * D], gtau[D * D];
#pragma unroll
        for (int i = 0; i < D * D; ++i) {
          gtau[i] = -c.ks * c.dx * gaff[i];
          gnF[i] = valid ? s.aF[i * P + p] : R(0);
        }
        const R gact = K::stress_adj(c, nF, m >= 0, am, fb, gtau, gnF);
        {
          const unsigned full = 0xffffffffu;
          const int m0 = __shfl_sync(full, m, 0);
          R* ga_e = a.gact + ((size_t)f * c.E + e) * c.M;
          if (__all_sync(full, m == m0)) {
            R sum = gact;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(full, sum, o);
            if (lane == 0 && m0 >= 0) atomicAdd(ga_e + m0, sum);
          } else if (m >= 0) {
            atomicAdd(ga_e + m, gact);
          }
        }
#pragma unroll
        for (int d = 0; d < D; ++d) ax[d] = (valid ? s.ax[d * P + p] : R(0)) + gfx[d] * c.inv_dx + seed[d];
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
          for (int j = 0; j < D; ++j) {
            R accC = 0, accF = 0;
#pragma unroll
            for (int k = 0; k < D; ++k) {
              accC += gnF[i * D + k] * Fp[j * D + k];
              accF += ((k == i ? R(1) : R(0)) + c.dt * Cp[k * D + i]) * gnF[k * D + j];
            }
            aC[i * D + j] = c.mass * c.dx * gaff[i * D + j] + c.dt * accC;
            aFo[i * D + j] = accF;
          }
        if (f == 0) {
          if (valid) {
#pragma unroll
            for (int d = 0; d < D; ++d) {
              a.out_ax[d * EP + q] = ax[d];
              a.out_av[d * EP + q] = av[d];
            }
#pragma unroll
            for (int i = 0; i < D * D; ++i) {
              a.out_aC[i * EP + q] = aC[i];
              a.out_aF[i * EP + q] = aFo[i];
            }
          }
          continue;
        }
      } else {
#pragma unroll
        for (int d = 0; d < D; ++d) {
          ax[d] = seed[d];
          av[d] = 0;
        }
#pragma unroll
        for (int i = 0; i < D * D; ++i) aC[i] = aFo[i] = 0;
      }
      // ---- G2P^T of step f - 1
      R xh[D];
#pragma unroll
      for (int d = 0; d < D; ++d) xh[d] = ld(rh + d * EP + q);
      K::weights(xh, c.inv_dx, n, base, fx, w, dw);
      R gvt[D], gfx[D];
#pragma unroll
      for (int i = 0; i < D; ++i) {
        gvt[i] = av[i] + c.dt * ax[i];
        gfx[i] = 0;
      }
      const R s4 = R(4) * c.inv_dx;
      const WarpRuns runs = warp_runs<D>(valid, base);
      const int slot = scatter_slot<R, D, D>(s.sc, runs, valid, nodes, a.cap, f & 1, small_node<D>(n, base), base[0]);
#pragma unroll
      for (int nq = 0; nq < K::NN; ++nq) {
        int o[D], I[D];
        K::offs(nq, o);
        const R wt = K::wgt(w, o);
        R dwt[D], dp[D];
        K::dwgt(w, dw, o, dwt);
#pragma unroll
        for (int d = 0; d < D; ++d) {
          dp[d] = (R)o[d] - fx[d];
          I[d] = base[d] + o[d];
        }
        const int node = small_node<D>(n, I);
        const V4<R> g4 = s.gv[node];
        const R g[3] = {g4.x, g4.y, g4.z};
        R gw = 0, sc[D];
#pragma unroll
        for (int i = 0; i < D; ++i) {
          R gGC = 0;
#pragma unroll
          for (int j = 0; j < D; ++j) gGC += aC[i * D + j] * dp[j];
          sc[i] = valid ? wt * (gvt[i] + s4 * gGC) : R(0);
          gw += g[i] * (gvt[i] + s4 * gGC);
        }
#pragma unroll
        for (int j = 0; j < D; ++j) {
          R acc = 0;
#pragma unroll
          for (int i = 0; i < D; ++i) acc += aC[i * D + j] * g[i];
          gfx[j] -= s4 * wt * acc;
        }
#pragma unroll
        for (int d = 0; d < D; ++d) gfx[d] += gw * dwt[d];
        scatter_add<R, D, D>(s.sc, runs, valid, nodes, a.cap, slot, nq, node, sc);
      }
      if (valid) {
#pragma unroll
        for (int d = 0; d < D; ++d) s.ax[d * P + p] = ax[d] + gfx[d] * c.inv_dx;
#pragma unroll
        for (int i = 0; i < D * D; ++i) s.aF[i * P + p] = aFo[i];
      }
    }
    __syncthreads();
  }
}

}  // namespace mpm
}  // namespace cls
