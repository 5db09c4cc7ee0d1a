// ms_cluster.cuh -- the fused segment kernels with one thread-block cluster per
// environment, for launches that leave most of the GPU idle when an environment
// runs in a single CTA.
//
// A substep of one env is a chain of short phases (observables, controller
// layers, spring gather), each bound by the latency and the load bandwidth of
// one SM.  Here the C CTAs of a cluster split every phase -- the rows (forward)
// and columns (adjoint) of the controller's layers, and the vertices -- and
// exchange the results by storing them into all C CTAs' shared memory, with
// one cluster barrier per exchange:
//   forward:  layer outputs (one exchange per layer), new x and v
//   reverse:  d v_inc, d outputs (each output's owner adds what the vertices'
//             CTAs send), partial sums of the output layer's transposed product,
//             hidden layers' dz, the centre's adjoint
// Every CTA holds the positions and velocities of the whole env, so the springs
// of its own vertices read them from its own shared memory; their incidence
// records are loaded into shared memory once per work item.  The forward pass
// computes the same bits as ms_forward_kernel at the same block size: rows,
// vertices and the centre are summed in the same order, whoever sums them.
//
// Measured on B200, one CTA per env against clusters of 8: 24 random lattices of
// 50-1974 vertices, 90 substeps over four segments, first pass 10.3 -> 2.3 ms,
// recompute 4.3 -> 0.85, reverse 12.1 -> 3.5; one quadruped, 101 substeps, 0.91
// -> 0.64 ms.  What bounds a small robot now is the instruction count of each
// phase (about 1 k per warp and substep) and, with L layers, L + 1 cluster barriers
// forward and L + 2 in reverse of ~0.5 us each.
#pragma once
#include <type_traits>

#include "ms_cluster_host.h"
#include "ms_segment.cuh"

namespace cls {

constexpr int kClusterMaxThreads = 512;

namespace cl {

__device__ __forceinline__ void copy16(void* dst_shared, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_shared);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// n bytes (a multiple of 16, both sides 16-byte aligned) by all threads
__device__ __forceinline__ void copy_bytes(void* dst, const void* src, int n) {
  for (int q = 16 * threadIdx.x; q < n; q += 16 * blockDim.x)
    copy16(static_cast<char*>(dst) + q, static_cast<const char*>(src) + q);
}

struct Carver {
  char* base;
  size_t off;
  __host__ __device__ Carver(char* b) : base(b), off(0) {}
  __host__ __device__ char* take(size_t bytes) {
    char* p = base + off;
    off += (bytes + 127) & ~size_t(127);
    return p;
  }
};

// incidence records of the CTA's own vertices in shared memory
template <typename R>
struct Incidence {
  int* ptr;        // own + 1 row starts, relative to the first own record
  int4* i;         // FP32: packed records; FP64: index records (caps.inc > 0)
  V4<R>* f;        // FP64: constants
};

template <typename R>
struct FwdShared {
  V4<R>* x[2];
  V4<R>* v[2];
  R* ain;
  R* hid;          // kMaxLayers - 1 rows of caps.h
  R* out;
  R* red;          // 4 x 32
  unsigned char* head;
  Incidence<R> inc;
};

template <typename R>
__host__ __device__ inline size_t carve(char* base, const ClusterCaps& c, FwdShared<R>* s) {
  Carver m(base);
  FwdShared<R> z;
  for (int b = 0; b < 2; ++b) {
    z.x[b] = (V4<R>*)m.take(sizeof(V4<R>) * c.n);
    z.v[b] = (V4<R>*)m.take(sizeof(V4<R>) * c.n);
  }
  z.ain = (R*)m.take(sizeof(R) * c.p0);
  z.hid = (R*)m.take(sizeof(R) * (kMaxLayers - 1) * c.h);
  z.out = (R*)m.take(sizeof(R) * c.o);
  z.red = (R*)m.take(sizeof(R) * 4 * 33);
  z.head = (unsigned char*)m.take(c.n);
  z.inc.ptr = (int*)m.take(sizeof(int) * (c.own + 1));
  z.inc.i = (int4*)m.take(sizeof(int4) * c.inc);
  z.inc.f = sizeof(R) == 8 ? (V4<R>*)m.take(sizeof(V4<R>) * c.inc) : nullptr;
  if (s) *s = z;
  return m.off;
}

template <typename R>
struct RevShared {
  V4<R>* x;
  V4<R>* v;        // of the substep being reversed, whole env
  V4<R>* gvi;      // d v_inc, whole env
  V4<R>* gx;
  V4<R>* gv;       // adjoint state of the own vertices
  V4<R>* vi;       // v_inc of the own vertices
  V4<R>* xo;       // x of the own vertices
  R* z;            // output layer's pre-activations
  R* out;          // controller outputs
  R* gout;         // d outputs of the own slice
  R* actd;         // activation derivative of the own slice
  R* part;         // [C][h] partial sums of the output layer's transposed product
  R* dz;           // [kMaxLayers - 1][h] dz of the hidden layers
  V4<R>* scratch;  // one per thread
  R* gin;          // d input positions of the own vertices
  R* gc;           // [C + 1][4] centre adjoint: the CTAs' partial sums, the velocity loss's seed
  R* red;          // kRed
  Incidence<R> inc;
};

template <typename R>
__host__ __device__ inline size_t carve(char* base, const ClusterCaps& c, int C, int threads, RevShared<R>* s) {
  Carver m(base);
  RevShared<R> z;
  z.x = (V4<R>*)m.take(sizeof(V4<R>) * c.n);
  z.v = (V4<R>*)m.take(sizeof(V4<R>) * c.n);
  z.gvi = (V4<R>*)m.take(sizeof(V4<R>) * c.n);
  z.gx = (V4<R>*)m.take(sizeof(V4<R>) * c.own);
  z.gv = (V4<R>*)m.take(sizeof(V4<R>) * c.own);
  z.vi = (V4<R>*)m.take(sizeof(V4<R>) * c.own);
  z.xo = (V4<R>*)m.take(sizeof(V4<R>) * c.own);
  z.z = (R*)m.take(sizeof(R) * c.o);
  z.out = (R*)m.take(sizeof(R) * c.o);
  z.gout = (R*)m.take(sizeof(R) * c.oslice);
  z.actd = (R*)m.take(sizeof(R) * c.oslice);
  z.part = (R*)m.take(sizeof(R) * c.h * C);
  z.dz = (R*)m.take(sizeof(R) * (kMaxLayers - 1) * c.h);
  z.scratch = (V4<R>*)m.take(sizeof(V4<R>) * threads);
  z.gin = (R*)m.take(sizeof(R) * (3 * c.own + 4));
  z.gc = (R*)m.take(sizeof(R) * 4 * (C + 1));
  z.red = (R*)m.take(sizeof(R) * kRed);
  z.inc.ptr = (int*)m.take(sizeof(int) * (c.own + 1));
  z.inc.i = (int4*)m.take(sizeof(int4) * c.inc);
  z.inc.f = sizeof(R) == 8 ? (V4<R>*)m.take(sizeof(V4<R>) * c.inc) : nullptr;
  if (s) *s = z;
  return m.off;
}

// row starts and records of vertices [v0, v1)
template <typename R>
__device__ __forceinline__ void load_incidence(const MsArgs<R>& a, const RobotDesc& rb, const ClusterCaps& c,
                                               const Incidence<R>& inc, int v0, int v1) {
  const int* ptr = a.inc_ptr + rb.ptr_off;
  const int q0 = ptr[v0], nq = ptr[v1] - q0;
  for (int i = threadIdx.x; i <= v1 - v0; i += blockDim.x) inc.ptr[i] = ptr[v0 + i] - q0;
  if (c.inc == 0) return;
  for (int q = threadIdx.x; q < nq; q += blockDim.x) {
    if constexpr (sizeof(R) == 4) {
      inc.i[q] = a.inc_p[rb.inc_off + q0 + q];
    } else {
      inc.i[q] = a.inc_i[rb.inc_off + q0 + q];
      inc.f[q] = a.inc_f[rb.inc_off + q0 + q];
    }
  }
}

// record q of the own vertices (counted from the first own record q0)
template <typename R>
__device__ __forceinline__ Inc<R> get_inc(const MsArgs<R>& a, const RobotDesc& rb, const ClusterCaps& c,
                                          const Incidence<R>& inc, int q0, int q, unsigned long long pol) {
  if (c.inc == 0) return load_inc<R>(a, rb, q0 + q, pol);
  Inc<R> r;
  const int4 p = inc.i[q];
  if constexpr (sizeof(R) == 4) {
    r.other = p.x & 0x7fff;
    r.side = (p.x >> 15) & 1;
    r.out = (int)(((unsigned)p.x) >> 16) - 1;
    r.l0 = __int_as_float(p.y);
    r.k = __int_as_float(p.z);
    r.coef = __int_as_float(p.w);
  } else {
    const V4<R> f = inc.f[q];
    r.other = p.x; r.side = p.y; r.out = p.w;
    r.l0 = f.x; r.k = f.y; r.coef = f.z;
  }
  return r;
}

// Centre of the env over the block, in block_sum<R, 3>'s order (strided thread
// sums, butterfly, warps in turn), with one barrier: after it every warp adds
// the warps' sums itself, lane m those of component m.
template <typename R>
__device__ __forceinline__ void block_center(R (&c)[3], R* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c[m] += __shfl_xor_sync(0xffffffffu, c[m], o);
  }
  if (lane == 0) {
#pragma unroll
    for (int m = 0; m < 3; ++m) red[m * 33 + wid] = c[m];
  }
  __syncthreads();
  R s = 0;
  if (lane < 3)
    for (int w = 0; w < nw; ++w) s += red[lane * 33 + w];
#pragma unroll
  for (int m = 0; m < 3; ++m) c[m] = __shfl_sync(0xffffffffu, s, m);
}

// Height, upper height, heading and centre of t into the observables, by one
// warp: compute_height / compute_rotation (solver_mass_spring.py:158-192).
template <typename R>
__device__ __forceinline__ void observe(const MsArgs<R>& a, const RobotDesc& rb, const EnvDesc& ed, const V4<R>* x,
                                        unsigned char* head, const R c[3], int e, int t, R& hprev) {
  const int lane = threadIdx.x & 31, N = rb.n_v;
  const bool heading = rb.robot_id != 100;
  R lo = R(10), hi = R(-10), h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = lane; i < N; i += 32) {
    const V4<R> p = x[i];
    lo = fmin(lo, p.y);
    hi = fmax(hi, p.y);
    if (heading) {
      if (t == 0) {
        const unsigned char f = p.x < c[0] ? 1 : 0;
        head[i] = f;
        a.head[ed.v_off + i] = f;
      }
      if (head[i]) { h[0] += p.x; h[1] += p.y; h[2] += p.z; h[3] += R(1); }
      else { h[4] += p.x; h[5] += p.y; h[6] += p.z; h[7] += R(1); }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
#pragma unroll
    for (int m = 0; m < 8; ++m) h[m] += __shfl_xor_sync(0xffffffffu, h[m], o);
  }
  R d0, d2;
  if (heading) {
    d0 = -h[0] * h[7] + h[4] * h[3];
    d2 = -h[2] * h[7] + h[6] * h[3];
  } else {
    const V4<R> p = x[rb.rot_idx[0]], q = x[rb.rot_idx[1]], u = x[rb.rot_idx[2]], w = x[rb.rot_idx[3]];
    d0 = p.x + q.x - u.x - w.x;
    d2 = p.z + q.z - u.z - w.z;
  }
  const R hh = (t % a.jump_period == 0) ? lo : fmax(hprev, lo);
  hprev = hh;
  if (lane == 0) {
    const size_t o = (size_t)t * a.n_envs + e;
    V4<R> cc; cc.x = c[0]; cc.y = c[1]; cc.z = c[2]; cc.w = 0;
    a.obs_center[o] = cc;
    a.obs_height[o] = hh;
    a.obs_upper[o] = hi;
    a.obs_rot[o] = datan2<R>(d2, d0);
  }
}

// Rows [lo, hi) of one layer, y = act(W x + b), by warps `wid` of `nw`, RB rows
// at a time; each row is summed in dense_forward's order (lane l: columns 4 l +
// 128 k, then the butterfly, halving the rows a lane holds while there are
// several).  y goes to all C CTAs' buffers, z to the record.
template <typename R, int RB>
__device__ __forceinline__ void layer_rows(const R* __restrict__ W, int pitch, int lo, int hi,
                                           const R* __restrict__ bias, const R* xin, R* y, R* zrec, int act, int wid,
                                           int nw, int C) {
  const int lane = threadIdx.x & 31;
  const int n4 = pitch >> 2;
  const V4<R>* x4 = reinterpret_cast<const V4<R>*>(xin);
  constexpr int UN = RB >= 8 ? 2 : (RB >= 4 ? 4 : 8);
  for (int i0 = lo + wid * RB; i0 < hi; i0 += nw * RB) {
    const V4<R>* w4[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) w4[r] = reinterpret_cast<const V4<R>*>(W + (size_t)(i0 + r < hi ? i0 + r : i0) * pitch);
    R s[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) s[r] = 0;
#pragma unroll UN
    for (int j = lane; j < n4; j += 32) {
      const V4<R> xv = x4[j];
      V4<R> wv[RB];
#pragma unroll
      for (int r = 0; r < RB; ++r) wv[r] = ldg4<R>(w4[r] + j);
#pragma unroll
      for (int r = 0; r < RB; ++r)
        s[r] += wv[r].x * xv.x + wv[r].y * xv.y + wv[r].z * xv.z + wv[r].w * xv.w;
    }
    // butterfly; while a lane holds several rows, it keeps half of them and
    // takes the partner lane's sums of those
    int row = 0, o = 16;
#pragma unroll
    for (int n = RB; n > 1; n >>= 1, o >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < n / 2; ++k) {
        const R give = up ? s[k] : s[k + n / 2], keep = up ? s[k + n / 2] : s[k];
        s[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
      row += up ? n / 2 : 0;
    }
    for (; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
    const int i = i0 + row;
    if (i < hi) {
      constexpr int G = 32 / RB;       // lanes that hold this row
      const int g = lane & (G - 1);
      const R v = act_f<R>(act, s[0] + bias[i]);
      if (zrec && g == 0) zrec[i] = s[0];
      for (int r = g; r < C; r += G) *peer(y + i, r) = v;
    }
  }
}

template <typename R>
__device__ __forceinline__ void layer(const R* W, int pitch, int lo, int hi, const R* bias, const R* xin, R* y, R* zrec,
                                      int act, int wid, int nw, int C) {
  const int n = hi - lo;
  if (n <= nw) layer_rows<R, 1>(W, pitch, lo, hi, bias, xin, y, zrec, act, wid, nw, C);
  else if (n <= 2 * nw) layer_rows<R, 2>(W, pitch, lo, hi, bias, xin, y, zrec, act, wid, nw, C);
  else if (n <= 4 * nw) layer_rows<R, 4>(W, pitch, lo, hi, bias, xin, y, zrec, act, wid, nw, C);
  else layer_rows<R, 8>(W, pitch, lo, hi, bias, xin, y, zrec, act, wid, nw, C);
}

// Split of a transposed product's G column groups and nrows rows over the
// block: slices of rows, and this thread's group and first row (tid = r0 G + g).
// Planned once per work item and layer: the divisions are slow against a phase.
struct ColumnSplit {
  int slices, g, r0;
};
__device__ __forceinline__ ColumnSplit column_split(int G, int nrows) {
  ColumnSplit c;
  c.slices = G > 0 ? (int)blockDim.x / G : 1;
  if (c.slices > 32) c.slices = 32;
  if (c.slices > nrows) c.slices = nrows;
  c.r0 = G > 0 ? (int)threadIdx.x / G : 0;
  c.g = (int)threadIdx.x - c.r0 * G;
  return c;
}

// out(g, sum_i W[i][4 g .. 4 g + 3] d[i]) for the column groups g0 <= g < g0 + G
// of an nrows-row matrix; scratch: one V4 per thread.  Threads split the rows
// when there are fewer groups than threads.  Ends with the sums given to out
// (by one thread each); the caller synchronises.
template <typename R, typename Out>
__device__ __forceinline__ void columns(const R* __restrict__ W, int pitch, int nrows, int g0, int G,
                                        const ColumnSplit& cs, const R* d, V4<R>* scratch, Out out) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int slices = cs.slices;
  if (slices <= 1) {
    for (int g = tid; g < G; g += nt) {
      V4<R> s;
      s.x = s.y = s.z = s.w = 0;
#pragma unroll 8
      for (int i = 0; i < nrows; ++i) {
        const V4<R> w = ldg4<R>(reinterpret_cast<const V4<R>*>(W + (size_t)i * pitch) + g0 + g);
        const R di = d[i];
        s.x += w.x * di; s.y += w.y * di; s.z += w.z * di; s.w += w.w * di;
      }
      out(g, s);
    }
    return;
  }
  if (cs.r0 < slices) {
    V4<R> s;
    s.x = s.y = s.z = s.w = 0;
    const V4<R>* w0 = reinterpret_cast<const V4<R>*>(W) + g0 + cs.g;
    const int p4 = pitch >> 2;
#pragma unroll 8
    for (int i = cs.r0; i < nrows; i += slices) {
      const V4<R> w = ldg4<R>(w0 + (size_t)i * p4);
      const R di = d[i];
      s.x += w.x * di; s.y += w.y * di; s.z += w.z * di; s.w += w.w * di;
    }
    scratch[tid] = s;
  }
  __syncthreads();
  if (tid < G) {
    V4<R> s = scratch[tid];
#pragma unroll 4
    for (int r = 1; r < slices; ++r) {
      const V4<R> p = scratch[r * G + tid];
      s.x += p.x; s.y += p.y; s.z += p.z; s.w += p.w;
    }
    out(tid, s);
  }
}

}  // namespace cl

// Segment [t_begin, t_end) of the launch's n_items envs, one cluster each
// (FwdMode bits and windows as ms_forward_kernel's).
template <typename R>
__global__ void __launch_bounds__(kClusterMaxThreads, 1)
ms_cluster_forward_kernel(MsArgs<R> a, ClusterCaps cap, int t_begin0, int t_end0, int mode, int src_slot0) {
  extern __shared__ __align__(256) char smem_raw[];
  __shared__ RobotDesc rb;
  __shared__ EnvDesc ed;
  const int C = (int)cl::size(), rank = (int)cl::rank();
  const int item = blockIdx.x / C;
  dependents_launch();  // the single-CTA launch of the lighter envs, if there is one
  if (item >= a.n_items) return;
  cl::FwdShared<R> s;
  cl::carve<R>(smem_raw, cap, &s);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  const int e = a.order[item];
  int t_begin = t_begin0, t_end = t_end0, src_slot = src_slot0;
  if (a.win) {
    const int4 w = a.win[e];
    t_begin = w.x; t_end = w.y; src_slot = w.z;
  }
  load_descs(a, e, rb, ed);
  const int N = rb.n_v, L = rb.n_layers, nout = rb.n_out;
  const int v0 = cluster_cut(N, kVertexUnit, rank, cap.log2c), v1 = cluster_cut(N, kVertexUnit, rank + 1, cap.log2c);
  const int q0 = a.inc_ptr[rb.ptr_off + v0];
  {
    const V4<R>* cx = a.ckpt_x + (size_t)src_slot * a.v_total + ed.v_off;
    const V4<R>* cv = a.ckpt_v + (size_t)src_slot * a.v_total + ed.v_off;
    for (int i = tid; i < N; i += nt) { s.x[0][i] = cx[i]; s.v[0][i] = cv[i]; }
    for (int i = tid; i < (kMaxLayers - 1) * cap.h; i += nt) s.hid[i] = 0;
    if ((mode & FWD_OBS) && t_begin > 0 && rb.robot_id != 100)
      for (int i = tid; i < N; i += nt) s.head[i] = a.head[ed.v_off + i];
    cl::load_incidence<R>(a, rb, cap, s.inc, v0, v1);
  }
  R hprev = 0;
  if ((mode & FWD_OBS) && t_begin > 0) hprev = a.obs_height[(size_t)(t_begin - 1) * a.n_envs + e];
  // sine and goal columns of the input, loaded one substep ahead of their use
  // (the velocity goals' division comes with the use, not with the load)
  const int p0 = rb.pos_pad, nc = rb.n_c, pitch0 = rb.pitch[0];
  const R invN = R(1) / R(N);
  auto tail = [&](int q, int t) {
    return q < p0 + a.n_sin ? a.sin_table[(size_t)t * a.n_sin + (q - p0)]
                            : goal_value<R>(a, q - p0 - a.n_sin, (size_t)t * a.n_envs + e);
  };
  const int qpre = p0 + tid;
  const R* src = nullptr;   // this thread's tail column: its value at t is src[t step]
  size_t step = 0;
  bool speed = false;
  if (qpre < p0 + a.n_sin) {
    src = a.sin_table + tid;
    step = a.n_sin;
  } else if (qpre < nc) {
    int g = qpre - p0 - a.n_sin;
    step = a.n_envs;
    if (a.dup_v > 0 && g < 2) {
      src = g == 0 ? &a.tv[e].x : &a.tv[e].z;
      step = 4 * (size_t)a.n_envs;
      speed = true;
    } else {
      g -= a.dup_v > 0 ? 2 : 0;
      if (a.dup_h > 0 && g == 0) src = a.th + e;
      else src = a.tc + e;
    }
  }
  R pre = (src && t_begin < t_end) ? src[t_begin * step] : R(0);
  int cur = 0, kmod = t_begin % a.K;
  // this CTA's rows of every layer
  __shared__ int s_lo[kMaxLayers], s_hi[kMaxLayers];
  if (tid < L) {
    s_lo[tid] = cluster_cut(rb.width[tid + 1], 1, rank, cap.log2c);
    s_hi[tid] = cluster_cut(rb.width[tid + 1], 1, rank + 1, cap.log2c);
  }
  const unsigned long long pol = policy_evict_last();
  cl::sync();  // every CTA is there and loaded before the first store into a peer
  for (int t = t_begin; t < t_end; ++t) {
    const V4<R>* x = s.x[cur];
    const V4<R>* v = s.v[cur];
    int kk = t - t_begin, mode_t = mode;
    if ((mode & FWD_RECTAIL) && t >= a.rec_from) {
      mode_t |= FWD_RECORD;
      kk = t - a.rec_from;
    }
    // ---- checkpoint, records and trajectory of the own vertices
    if ((mode & FWD_CKPT) && t > t_begin && kmod == 0) {
      V4<R>* cx = a.ckpt_x + (size_t)(t / a.K) * a.v_total + ed.v_off;
      V4<R>* cv = a.ckpt_v + (size_t)(t / a.K) * a.v_total + ed.v_off;
      bool bad = false;
      for (int i = v0 + tid; i < v1; i += nt) {
        cx[i] = x[i]; cv[i] = v[i];
        bad |= !(finite(x[i].x) && finite(x[i].y) && finite(x[i].z));
      }
      if (bad) atomicOr(a.status, ERR_NONFINITE);
    }
    if (mode_t & FWD_RECORD) {
      V4<R>* rx = a.rec_x + (size_t)kk * a.v_total + ed.v_off;
      V4<R>* rv = a.rec_v + (size_t)kk * a.v_total + ed.v_off;
      for (int i = v0 + tid; i < v1; i += nt) { rx[i] = x[i]; rv[i] = v[i]; }
    }
    if ((mode & FWD_OBS) && a.x_full) {
      V4<R>* xf = a.x_full + (size_t)t * a.v_total + ed.v_off;
      for (int i = v0 + tid; i < v1; i += nt) xf[i] = x[i];
    }
    if (mode & FWD_REPLAY) {
      // controller outputs from the recorded pre-activations, in every CTA
      const int lo = L - 1;
      const R* zr = a.rec_z + a.z_base[lo] + (size_t)kk * a.z_total[lo] + ed.z_off[lo];
      const R* bo = a.bias + rb.b_off[lo];
      for (int o = tid; o < nout; o += nt) s.out[o] = act_f<R>(a.act_out, zr[o] + bo[o]);
      __syncthreads();
    } else {
      const bool rec_ctrl = (mode_t & FWD_RECORD) || (mode & FWD_RECCTRL);
      const int kc = (mode & FWD_RECCTRL) ? t : kk;
      // ---- centre (solver_mass_spring.py:150-156), nn_input (taichi_env.py:149-183)
      R c[3] = {0, 0, 0};
      for (int i = tid; i < N; i += nt) {
        const V4<R> p = x[i];
        c[0] += p.x * invN; c[1] += p.y * invN; c[2] += p.z * invN;
      }
      cl::block_center<R>(c, s.red);
      R* rin = rec_ctrl ? a.rec_in + (size_t)kc * a.in_total + ed.in_off : nullptr;
      for (int i = tid; i < N; i += nt) {
        const V4<R> p = x[i];
        const R u0 = (p.x - c[0]) / R(0.2), u1 = (p.y - c[1]) / R(0.2), u2 = (p.z - c[2]) / R(0.2);
        s.ain[3 * i] = u0; s.ain[3 * i + 1] = u1; s.ain[3 * i + 2] = u2;
        if (rin && i >= v0 && i < v1) { rin[3 * i] = u0; rin[3 * i + 1] = u1; rin[3 * i + 2] = u2; }
      }
      for (int q = 3 * N + tid; q < pitch0; q += nt) {  // padding and what `pre` does not reach
        if (q >= p0 && q < nc && q - p0 < nt) continue;
        const R val = (q >= p0 && q < nc) ? tail(q, t) : R(0);
        s.ain[q] = val;
        if (rin && rank == 0 && q < nc) rin[q] = val;
      }
      if (src) {
        const R val = speed ? pre / a.max_speed : pre;
        s.ain[qpre] = val;
        if (rin && rank == 0) rin[qpre] = val;
        if (t + 1 < t_end) pre = src[(size_t)(t + 1) * step];
      }
      __syncthreads();
      // ---- MLP (nn.py:130-146), the layers' rows split over the CTAs.  The
      // last warp of the last CTA takes the observables instead: it arrives at
      // the first layer's barrier before it starts on them
      const bool observer = (mode & FWD_OBS) && rank == C - 1;
      const int nwl = observer ? nw - 1 : nw;
      for (int l = 0; l < L; ++l) {
        if (wid < nwl) {
          cl::layer<R>(a.w + rb.w_off[l], rb.pitch[l], s_lo[l], s_hi[l], a.bias + rb.b_off[l],
                       l == 0 ? s.ain : s.hid + (l - 1) * cap.h, l == L - 1 ? s.out : s.hid + l * cap.h,
                       rec_ctrl ? a.rec_z + a.z_base[l] + (size_t)kc * a.z_total[l] + ed.z_off[l] : nullptr,
                       l == L - 1 ? a.act_out : a.act_hidden, wid, nwl, C);
          cl::arrive();
        } else {
          cl::arrive();
          if (l == 0) cl::observe<R>(a, rb, ed, x, s.head, c, e, t, hprev);
        }
        cl::wait();
      }
    }
    if ((mode & FWD_OBS) && a.act_full && rank == 0) {
      R* af = a.act_full + (size_t)t * a.z_total[L - 1] + ed.z_off[L - 1];
      for (int o = tid; o < nout; o += nt) af[o] = s.out[o];
    }
    // ---- apply_spring_force and advance_toi of the own vertices: a half-warp
    // per vertex as in gather_vinc_all; its lanes advance the vertex and
    // lane r stores it to CTA r
    {
      V4<R>* rec = (mode_t & FWD_RECORD) ? a.rec_vinc + (size_t)kk * a.v_total + ed.v_off : nullptr;
      const int l16 = lane & 15, half = lane >> 4, stride = nw * 2;
      V4<R>* xn = s.x[cur ^ 1];
      V4<R>* vn = s.v[cur ^ 1];
      auto vertices = [&](int vb0, auto width) {
        constexpr int U = decltype(width)::value;
        R sum[U][3];
        V4<R> xi[U], vi[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int i = vb0 + half + k * stride;
          sum[k][0] = sum[k][1] = sum[k][2] = 0;
          if (i < v1) {
            xi[k] = x[i]; vi[k] = v[i];
            const int end = s.inc.ptr[i - v0 + 1];
            for (int q = s.inc.ptr[i - v0] + l16; q < end; q += 16)
              accumulate_incidence<R>(a, cl::get_inc<R>(a, rb, cap, s.inc, q0, q, pol), xi[k], vi[k], x, v, s.out,
                                      sum[k][0], sum[k][1], sum[k][2]);
          }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
#pragma unroll
          for (int k = 0; k < U; ++k)
#pragma unroll
            for (int m = 0; m < 3; ++m) sum[k][m] += __shfl_xor_sync(0xffffffffu, sum[k][m], o);
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
          const int i = vb0 + half + k * stride;
          if (i < v1) {
            V4<R> vc; vc.x = sum[k][0]; vc.y = sum[k][1]; vc.z = sum[k][2]; vc.w = 0;
            if (rec && l16 == 0) rec[i] = vc;
            advance_vertex<R>(a, xi[k], vi[k], vc);
            if (l16 < C) {
              *cl::peer(xn + i, l16) = xi[k];
              *cl::peer(vn + i, l16) = vi[k];
            }
          }
        }
      };
      // two vertices per half-warp at a time while there are that many
      int vb0 = v0 + wid * 2;
      for (; vb0 + stride < v1; vb0 += 2 * stride) vertices(vb0, std::integral_constant<int, 2>());
      if (vb0 < v1) vertices(vb0, std::integral_constant<int, 1>());
    }
    cl::sync();
    cur ^= 1;
    kmod = kmod + 1 == a.K ? 0 : kmod + 1;
  }
  // ---- state after the last substep
  const V4<R>* x = s.x[cur];
  const V4<R>* v = s.v[cur];
  if ((mode & FWD_CKEND) && t_end % a.K == 0 && t_end > t_begin) {
    V4<R>* cx = a.ckpt_x + (size_t)(t_end / a.K) * a.v_total + ed.v_off;
    V4<R>* cv = a.ckpt_v + (size_t)(t_end / a.K) * a.v_total + ed.v_off;
    for (int i = v0 + tid; i < v1; i += nt) { cx[i] = x[i]; cv[i] = v[i]; }
  }
  if (mode & FWD_OBS) {
    for (int i = v0 + tid; i < v1; i += nt) { a.fin_x[ed.v_off + i] = x[i]; a.fin_v[ed.v_off + i] = v[i]; }
    if (a.x_full && t_end < a.T) {
      V4<R>* xf = a.x_full + (size_t)t_end * a.v_total + ed.v_off;
      for (int i = v0 + tid; i < v1; i += nt) xf[i] = x[i];
    }
  }
}

// Adjoint of segment [t_begin, t_end), one cluster per env (arguments as
// ms_reverse_kernel's).
template <typename R>
__global__ void __launch_bounds__(kClusterMaxThreads, 1)
ms_cluster_reverse_kernel(MsArgs<R> a, ClusterCaps cap, int t_begin0, int t_end0, int last_seg0) {
  extern __shared__ __align__(256) char smem_raw[];
  __shared__ RobotDesc rb;
  __shared__ EnvDesc ed;
  const int C = (int)cl::size(), rank = (int)cl::rank();
  const int item = blockIdx.x / C;
  dependents_launch();  // the single-CTA launch of the lighter envs, if there is one
  if (item >= a.n_items) return;
  cl::RevShared<R> s;
  cl::carve<R>(smem_raw, cap, C, blockDim.x, &s);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  const int e = a.order[item];
  int t_begin = t_begin0, t_end = t_end0, last_seg = last_seg0;
  if (a.win) {
    const int4 w = a.win[e];
    t_begin = w.x; t_end = w.y; last_seg = w.w;
  }
  load_descs(a, e, rb, ed);
  const int N = rb.n_v, L = rb.n_layers, nout = rb.n_out;
  const int v0 = cluster_cut(N, kVertexUnit, rank, cap.log2c), v1 = cluster_cut(N, kVertexUnit, rank + 1, cap.log2c);
  const int nv = v1 - v0;
  const int q0 = a.inc_ptr[rb.ptr_off + v0];
  const int osl = (nout + C - 1) / C;   // outputs [rank osl, rank osl + osl) are this CTA's
  const int o0 = rank * osl < nout ? rank * osl : nout, o1 = o0 + osl < nout ? o0 + osl : nout;
  const R Br = R(rb.loss_envs), invN = R(1) / R(N);
  const unsigned osl_rcp = osl > 1 ? 0xffffffffu / (unsigned)osl + 1u : 0u;  // o / osl = umulhi(o, .) for o < 65536
  const bool whole_x = (a.loss_mask & (LOSS_HEIGHT | LOSS_CRAWL)) != 0;  // rev_post's extrema read all of x
  // splits of the transposed products: output layer, hidden layers' columns
  // (planned where they run: there is at most one in most controllers), inputs
  const int Gw = (rb.width[L - 1] + 3) >> 2, Gx = (3 * nv + 3) >> 2;
  const cl::ColumnSplit cs_out = cl::column_split(Gw, o1 - o0), cs_in = cl::column_split(Gx, rb.width[1]);
  const int hg0 = cluster_cut((rb.width[1] + 3) >> 2, 1, rank, cap.log2c);
  const int hg1 = cluster_cut((rb.width[1] + 3) >> 2, 1, rank + 1, cap.log2c);
  const cl::ColumnSplit cs_h1 = cl::column_split(hg1 - hg0, rb.width[L > 2 ? 2 : 1]);  // of layer 1
  const int rp = a.run_period, tp = a.turn_period, st_e = steps_of(a, e);
  __shared__ R s_rot[4];   // cos, sin of the heading goals at t - rp and t
  int* redi = reinterpret_cast<int*>(s.red + kRedInt);
  cl::load_incidence<R>(a, rb, cap, s.inc, v0, v1);
  R hcarry = last_seg ? R(0) : a.adj_h[e];
  for (int i = tid; i < nv; i += nt) {
    V4<R> gx, gv;
    if (last_seg) {
      R gxi[3] = {0, 0, 0}, gcd[3] = {0, 0, 0};
      if (a.x_full) {
        const V4<R> xi = a.x_full[(size_t)t_end * a.v_total + ed.v_off + v0 + i];
        seed_x_rotation_pose<R>(a, rb, ed, t_end, e, v0 + i, xi, Br, gxi, gcd);
      }
      gx.x = gxi[0]; gx.y = gxi[1]; gx.z = gxi[2]; gx.w = 0;
      gv.x = gv.y = gv.z = gv.w = 0;
    } else {
      gx = a.adj_x[ed.v_off + v0 + i];
      gv = a.adj_v[ed.v_off + v0 + i];
    }
    s.gx[i] = gx;
    s.gv[i] = gv;
  }
  for (int i = tid; i < osl; i += nt) s.gout[i] = 0;
  // records of substep t into shared memory (asynchronous copies)
  auto fetch = [&](int t) {
    const int kk = t - t_begin;
    const size_t ro = (size_t)kk * a.v_total + ed.v_off;
    cl::copy_bytes(s.x, a.rec_x + ro, (int)sizeof(V4<R>) * N);
    cl::copy_bytes(s.v, a.rec_v + ro, (int)sizeof(V4<R>) * N);
    cl::copy_bytes(s.vi, a.rec_vinc + ro + v0, (int)sizeof(V4<R>) * nv);
    cl::copy_bytes(s.z, a.rec_z + a.z_base[L - 1] + (size_t)kk * a.z_total[L - 1] + ed.z_off[L - 1],
                   (int)sizeof(R) * ((nout + 3) & ~3));
    cl::copy_commit();
  };
  if (t_begin < t_end) fetch(t_end - 1);
  const R* bout = a.bias + rb.b_off[L - 1];
  const unsigned long long pol = policy_evict_last();
  cl::sync();
  for (int t = t_end - 1; t >= t_begin; --t) {
    const int kk = t - t_begin;
    cl::copy_wait();
    __syncthreads();
    // ---- loads of the loss seeds, used at the end of the substep: the rotation
    // loss's other positions for the thread's first vertex, the centres, and
    // (two threads) the velocity loss's seed
    const bool on1 = (a.loss_mask & LOSS_ROTATION) && t >= 1 && t % tp > rp && t <= st_e && t < a.T;
    const int u = t + rp;
    const bool on2 = (a.loss_mask & LOSS_ROTATION) && u <= st_e && u < a.T && u % tp > rp;
    V4<R> xm, xp;
    xm.x = xm.y = xm.z = xm.w = 0;
    xp = xm;
    if (tid < nv) {
      if (on1) xm = a.x_full[(size_t)(t - rp) * a.v_total + ed.v_off + v0 + tid];
      if (on2) xp = a.x_full[(size_t)u * a.v_total + ed.v_off + v0 + tid];
    }
    V4<R> ct, cm, cp;
    ct.x = ct.y = ct.z = ct.w = 0;
    cm = cp = ct;
    if (on1 || on2) ct = obs_c(a, t, e);
    if (on1) cm = obs_c(a, t - rp, e);
    if (on2) cp = obs_c(a, u, e);
    R th = 0;
    if (tid < 2 && (tid == 0 ? on1 : on2)) th = a.th[(size_t)(tid == 0 ? t - rp : t) * a.n_envs + e];
    R gvel[3] = {0, 0, 0};
    if (rank == 0 && tid == 64 % nt) apply_center_velocity<R>(load_center_velocity<R>(a, t, e, Br), gvel);
    // ---- outputs; adjoint of advance_toi(t + 1) for the own vertices
    for (int o = tid; o < nout; o += nt) {
      const R u = s.z[o] + bout[o];
      s.out[o] = act_f<R>(a.act_out, u);
      if (o >= o0 && o < o1) s.actd[o - o0] = act_d<R>(a.act_out, u);
    }
    for (int i = tid; i < nv; i += nt) {
      const V4<R> x = s.x[v0 + i], v = s.v[v0 + i], vi = s.vi[i], gx1 = s.gx[i], gv1 = s.gv[i];
      s.xo[i] = x;
      V4<R> gx0, gv0, gvi;
      advance_adjoint<R>(a, x, v, vi, gx1, gv1, gx0, gv0, gvi);
      s.gx[i] = gx0;
      s.gv[i] = gv0;
      for (int r = 0; r < C; ++r) *cl::peer(s.gvi + v0 + i, r) = gvi;
    }
    if (tid < 2) {
      const R ang = th * R(72.) / R(180.) * R(3.1415926535);
      s_rot[2 * tid] = dcos<R>(ang);
      s_rot[2 * tid + 1] = dsin<R>(ang);
    }
    cl::sync();
    // ---- adjoint of apply_spring_force(t): half-warp per own vertex
    {
      const size_t o = (size_t)t * a.n_envs + e;
      const bool act_seed = (a.loss_mask & LOSS_ACTUATION) && t < st_e && a.th[o] < R(0.1 + 1e-4);
      const R lim = act_seed ? dpow_half<R>(dabs<R>(a.tv[o].x) / R(0.08)) : R(0);
      const R act_scale = act_seed ? R(10) / R(st_e) / Br / R(rb.n_s) : R(0);
      const int l16 = lane & 15, half = lane >> 4, stride = nw * 2;
      {
        for (int vb0 = wid * 2; vb0 < nv; vb0 += stride) {
          const int i = vb0 + half;
          R gxs[3] = {0, 0, 0}, gvs[3] = {0, 0, 0};
          if (i < nv) {
            const int end = s.inc.ptr[i + 1];
            for (int q = s.inc.ptr[i] + l16; q < end; q += 16) {
              const Inc<R> in = cl::get_inc<R>(a, rb, cap, s.inc, q0, q, pol);
              const int ia = in.side == 0 ? v0 + i : in.other, ib = in.side == 0 ? in.other : v0 + i;
              const R act = in.out >= 0 ? s.out[in.out] : R(0);
              const SpringAdj<R> g = spring_adjoint_terms<R>(a, s.x[ia], s.x[ib], s.v[ia], s.v[ib], s.gvi[ia],
                                                             s.gvi[ib], act, in.l0, in.k, in.coef);
              if (in.side == 0) {
                gxs[0] += g.gd0; gxs[1] += g.gd1; gxs[2] += g.gd2;
                gvs[0] += g.h0; gvs[1] += g.h1; gvs[2] += g.h2;
                if (in.out >= 0) {
                  const int owner = osl > 1 ? (int)__umulhi((unsigned)in.out, osl_rcp) : in.out;
                  atomicAdd(cl::peer(s.gout + (in.out - owner * osl), owner),
                            spring_gact<R>(g.gact, act, act_scale, lim, act_seed));
                }
              } else {
                gxs[0] -= g.gd0; gxs[1] -= g.gd1; gxs[2] -= g.gd2;
                gvs[0] -= g.h0; gvs[1] -= g.h1; gvs[2] -= g.h2;
              }
            }
          }
#pragma unroll
          for (int o = 8; o > 0; o >>= 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              gxs[c] += __shfl_xor_sync(0xffffffffu, gxs[c], o);
              gvs[c] += __shfl_xor_sync(0xffffffffu, gvs[c], o);
            }
          }
          if (l16 == 0 && i < nv) {
            V4<R> x = s.gx[i], w = s.gv[i];
            x.x += gxs[0]; x.y += gxs[1]; x.z += gxs[2];
            w.x += gvs[0]; w.y += gvs[1]; w.z += gvs[2];
            s.gx[i] = x;
            s.gv[i] = w;
          }
        }
      }
    }
    cl::sync();
    if (!whole_x && t > t_begin) fetch(t - 1);  // x, v, v_inc and z of t are not read any more
    // ---- dz of the own outputs; partial sums of the output layer's
    // transposed product over them, to all CTAs
    {
      R* dzr = a.rec_dz + a.z_base[L - 1] + (size_t)kk * a.z_total[L - 1] + ed.z_off[L - 1];
      for (int q = tid; q < o1 - o0; q += nt) {
        const R dz = s.gout[q] * s.actd[q];
        s.actd[q] = dz;
        s.gout[q] = 0;
        dzr[o0 + q] = dz;
      }
      __syncthreads();
      if (rank == 0 && tid == 64 % nt)
        for (int r = 0; r < C; ++r) {
          R* g = cl::peer(s.gc + 4 * C, r);
          g[0] = gvel[0]; g[1] = gvel[1]; g[2] = gvel[2];
        }
      cl::columns<R>(a.w + rb.w_off[L - 1] + (size_t)o0 * rb.pitch[L - 1], rb.pitch[L - 1], o1 - o0, 0, Gw, cs_out,
                     s.actd, s.scratch, [&](int g, const V4<R>& p) {
                       for (int r = 0; r < C; ++r)
                         *cl::peer(reinterpret_cast<V4<R>*>(s.part + rank * cap.h) + g, r) = p;
                     });
    }
    // pre-activations of the last hidden layer, ahead of the barrier
    const int wl = rb.width[L - 1];
    const size_t zo = a.z_base[L - 2] + (size_t)kk * a.z_total[L - 2] + ed.z_off[L - 2];
    const R uz = tid < wl ? a.rec_z[zo + tid] + a.bias[rb.b_off[L - 2] + tid] : R(0);
    cl::sync();
    {
      R* dzl = s.dz + (L - 2) * cap.h;
      for (int q = tid; q < wl; q += nt) {
        R d = s.part[q];
        for (int r = 1; r < C; ++r) d += s.part[r * cap.h + q];
        const R u = q < nt ? uz : a.rec_z[zo + q] + a.bias[rb.b_off[L - 2] + q];
        const R dz = d * act_d<R>(a.act_hidden, u);
        dzl[q] = dz;
        if ((q & (C - 1)) == rank) a.rec_dz[zo + q] = dz;
      }
      __syncthreads();
    }
    // ---- hidden layers: the columns split over the CTAs
    for (int l = L - 2; l >= 1; --l) {
      const int nin = rb.width[l], G = (nin + 3) >> 2;
      const int g0 = l == 1 ? hg0 : cluster_cut(G, 1, rank, cap.log2c);
      const int g1 = l == 1 ? hg1 : cluster_cut(G, 1, rank + 1, cap.log2c);
      const cl::ColumnSplit cs = l == 1 ? cs_h1 : cl::column_split(g1 - g0, rb.width[l + 1]);
      const size_t zi = a.z_base[l - 1] + (size_t)kk * a.z_total[l - 1] + ed.z_off[l - 1];
      R* dzl = s.dz + (l - 1) * cap.h;
      cl::columns<R>(a.w + rb.w_off[l], rb.pitch[l], rb.width[l + 1], g0, g1 - g0, cs, s.dz + l * cap.h, s.scratch,
                     [&](int g, const V4<R>& p) {
                       const int q = 4 * (g0 + g);
                       const R pv[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
                       for (int u = 0; u < 4; ++u) {
                         if (q + u >= nin) continue;
                         const R dz = pv[u] * act_d<R>(a.act_hidden, a.rec_z[zi + q + u] + a.bias[rb.b_off[l - 1] + q + u]);
                         a.rec_dz[zi + q + u] = dz;
                         for (int r = 0; r < C; ++r) *cl::peer(dzl + q + u, r) = dz;
                       }
                     });
      cl::sync();
    }
    // ---- first layer: the position columns of the own vertices
    cl::columns<R>(a.w + rb.w_off[0], rb.pitch[0], rb.width[1], 3 * v0 / 4, Gx, cs_in, s.dz, s.scratch,
                   [&](int g, const V4<R>& p) { reinterpret_cast<V4<R>*>(s.gin)[g] = p; });
    __syncthreads();
    // ---- nn_input, centre and loss seeds (rev_post), own vertices
    {
      R gc[3] = {0, 0, 0};
      const R krot = R(2) / R(40) / R(st_e);
      for (int i = tid; i < nv; i += nt) {
        const R g0 = s.gin[3 * i] / R(0.2), g1 = s.gin[3 * i + 1] / R(0.2), g2 = s.gin[3 * i + 2] / R(0.2);
        R gxi[3] = {g0, g1, g2};
        gc[0] -= g0; gc[1] -= g1; gc[2] -= g2;
        const V4<R> xi = s.xo[i];
        if (i >= nt) {
          if (on1) xm = a.x_full[(size_t)(t - rp) * a.v_total + ed.v_off + v0 + i];
          if (on2) xp = a.x_full[(size_t)u * a.v_total + ed.v_off + v0 + i];
        }
        if (on1) rotation_seed_late<R>(xi, ct, xm, cm, s_rot[0], s_rot[1], krot, gxi, gc);
        if (on2) rotation_seed_early<R>(xp, cp, xi, ct, s_rot[2], s_rot[3], krot, gxi, gc);
        pose_seed<R>(a, ed, t, e, v0 + i, xi, Br, gxi);
        V4<R> gx = s.gx[i];
        gx.x += gxi[0]; gx.y += gxi[1]; gx.z += gxi[2];
        s.gx[i] = gx;
      }
      cl::block_center<R>(gc, s.red);
      if (tid < 3 * C) {
        const int m = tid % 3;
        *cl::peer(s.gc + 4 * rank + m, tid / 3) = m == 0 ? gc[0] : (m == 1 ? gc[1] : gc[2]);
      }
      cl::sync();
      gc[0] = gc[1] = gc[2] = 0;
      for (int r = 0; r <= C; ++r) {
        gc[0] += s.gc[4 * r]; gc[1] += s.gc[4 * r + 1]; gc[2] += s.gc[4 * r + 2];
      }
      for (int i = tid; i < nv; i += nt) {
        V4<R> gx = s.gx[i];
        gx.x += gc[0] * invN; gx.y += gc[1] * invN; gx.z += gc[2] * invN;
        s.gx[i] = gx;
      }
    }
    // ---- running height and upper height: the extrema in every CTA, their
    // vertices' adjoint in the owner's
    if (whole_x) {
      const R gh = seed_height<R>(a, t, e, Br) + hcarry;
      const R gu = seed_upper<R>(a, t, e, Br);
      hcarry = 0;
      __syncthreads();
      if (gh != R(0)) {
        R lo = R(10); int li = -1;
        for (int i = tid; i < N; i += nt) {
          const R y = s.x[i].y;
          if (!(lo < y)) { lo = y; li = i; }
        }
        block_argext<R>(lo, li, true, s.red, redi);
        R gmin = gh;
        if (t % a.jump_period != 0) {
          const R prev = a.obs_height[(size_t)(t - 1) * a.n_envs + e];
          if (lo < prev) { hcarry = gh; gmin = 0; }
        }
        if (tid == 0 && li >= v0 && li < v1 && gmin != R(0)) s.gx[li - v0].y += gmin;
      }
      if (gu != R(0)) {
        R hi = R(-10); int hix = -1;
        for (int i = tid; i < N; i += nt) {
          const R y = s.x[i].y;
          if (!(y < hi)) { hi = y; hix = i; }
        }
        block_argext<R>(hi, hix, false, s.red, redi);
        if (tid == 0 && hix >= v0 && hix < v1) s.gx[hix - v0].y += gu;
      }
      __syncthreads();
      if (t > t_begin) fetch(t - 1);
    }
  }
  __syncthreads();
  for (int i = tid; i < nv; i += nt) {
    a.adj_x[ed.v_off + v0 + i] = s.gx[i];
    a.adj_v[ed.v_off + v0 + i] = s.gv[i];
  }
  if (tid == 0 && rank == 0) a.adj_h[e] = hcarry;
  cl::sync();  // no CTA leaves while a peer may still store into it
}

}  // namespace cls
