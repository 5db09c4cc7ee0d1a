// noalloc.cu -- cls_ms_advance_noalloc: mass-spring substeps that allocate no
// memory at all.
//
// Who needs this: callers that are not allowed to allocate device memory --
// code running under a fixed device-memory budget owned by someone else (a
// game or robotics runtime with its own allocator, a serving process whose
// memory pool is pre-sized), or code that must not create allocations while a
// larger system is capturing its own work.  cls_create allocates its buffers
// with cudaMalloc, so such callers cannot use a cls_sim handle.  This entry
// point takes every input and output as a caller-owned device pointer and keeps
// its one piece of scratch -- the per-vertex velocity increment v_inc that the
// spring forces accumulate into -- in a fixed array that is part of the
// library image.
//
// Limits and sharing rules:
//   * the scratch holds kScratchFloats floats (2^21 = 8 MiB): calls need
//     n_envs * n_vertices * 3 <= kScratchFloats and are rejected otherwise;
//   * every GPU that loads the library holds that 8 MiB until the process ends;
//   * robots whose springs fit in one CTA's shared memory (about 5000) need no
//     scratch: one launch runs all substeps (na_fused, na_slices).  Larger ones use the
//     array, and calls that overlap on the GPU race with each other there and
//     give wrong results; serialise them;
//   * each call clears the part it uses before the first substep, so nothing
//     left from an earlier call leaks into the result;
//   * a __device__ array's address belongs to a CUDA context, so the first
//     call in each context (the runtime's primary context of a device, or a
//     context the caller created and made current with the driver API) looks
//     up the array's device address (cudaGetSymbolAddress) with that context
//     current and keeps it keyed by the context's unique id (cuCtxGetId: ids
//     are never reused, so a context created after cudaDeviceReset or
//     cuCtxDestroy gets a fresh lookup); make that first call before any
//     stream capture in that context;
//   * spring endpoints must lie in [0, n_vertices); a spring whose endpoint
//     does not is skipped (it exerts no force), so a bad table never reads or
//     writes outside the env's rows;
//   * a CUDA error already pending when the call starts (from the caller's
//     earlier work) is left in place and reported as CLS_ERR_CUDA without
//     launching anything.
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "../../include/cls_b200.h"
#include "cls_context.h"
#include "ms_kernels.cuh"

namespace {

constexpr long long kScratchFloats = 1LL << 21;
constexpr int kMaxContexts = 64;

// v_inc scratch ([env][vertex][3]); in host code this name is only a handle
// for cudaGetSymbolAddress, never a usable address
static __device__ __align__(256) float g_vinc_scratch[kScratchFloats];

// the scratch's address per CUDA context, keyed by the context's unique id
struct ScratchEntry {
  unsigned long long ctx_id;
  void* addr;
};
ScratchEntry g_scratch[kMaxContexts] = {};
int g_scratch_used = 0, g_scratch_next = 0;
std::mutex g_scratch_mutex;

// The scratch's device address in the current context; on the first call in a
// context, cudaGetSymbolAddress (which also makes the device's primary context
// current when no context is) resolves it with that context current.
cudaError_t scratch_address(float** out) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  unsigned long long id = 0;
  if (!cls::current_ctx_id(&id)) return cudaErrorNotSupported;
  if (id) {
    for (int i = 0; i < g_scratch_used; ++i)
      if (g_scratch[i].ctx_id == id) {
        *out = static_cast<float*>(g_scratch[i].addr);
        return cudaSuccess;
      }
  }
  void* p = nullptr;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_vinc_scratch);
  if (e != cudaSuccess) return e;
  if (!p) return cudaErrorInvalidSymbol;
  if (!id) cls::current_ctx_id(&id);   // the lookup made the primary context current
  if (id) {
    int slot = g_scratch_used < kMaxContexts ? g_scratch_used++ : g_scratch_next;
    if (g_scratch_used == kMaxContexts) g_scratch_next = (slot + 1) % kMaxContexts;
    g_scratch[slot] = ScratchEntry{id, p};
  }
  *out = static_cast<float*>(p);
  return cudaSuccess;
}

void set_message(const cls_noalloc_advance* a, const char* msg) {
  if (a && a->error_message && a->error_capacity > 0)
    snprintf(a->error_message, (size_t)a->error_capacity, "%s", msg);
}

__global__ void na_clear(float* __restrict__ s, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    s[i] = 0.f;
}

// apply_spring_force (solver_mass_spring.py:86-105): one thread per (env,
// spring), impulses scattered into v_inc with atomics as the reference does
__global__ void na_spring(cls_noalloc_advance a, float* __restrict__ vinc) {
  const long long total = (long long)a.n_envs * a.n_springs;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    const int e = (int)(q / a.n_springs), s = (int)(q % a.n_springs);
    const int ia = a.spring_a[s], ib = a.spring_b[s];
    if (ia < 0 || ia >= a.n_vertices || ib < 0 || ib >= a.n_vertices) continue;
    const float* xe = a.x + (size_t)e * a.n_vertices * 3;
    const float* ve = a.v + (size_t)e * a.n_vertices * 3;
    cls::V4<float> xa, xb, va, vb;
    xa.x = xe[3 * ia]; xa.y = xe[3 * ia + 1]; xa.z = xe[3 * ia + 2]; xa.w = 0;
    xb.x = xe[3 * ib]; xb.y = xe[3 * ib + 1]; xb.z = xe[3 * ib + 2]; xb.w = 0;
    va.x = ve[3 * ia]; va.y = ve[3 * ia + 1]; va.z = ve[3 * ia + 2]; va.w = 0;
    vb.x = ve[3 * ib]; vb.y = ve[3 * ib + 1]; vb.z = ve[3 * ib + 2]; vb.w = 0;
    float imp[3];
    cls::spring_impulse<float>(xa, xb, va, vb, a.rest_length[s], a.stiffness[s], a.actuation_coef[s],
                               a.actuation[(size_t)e * a.n_springs + s], a.dt, a.dashpot_damping, imp);
    float* vi = vinc + (size_t)e * a.n_vertices * 3;
    for (int d = 0; d < 3; ++d) {
      atomicAdd(vi + 3 * ia + d, -imp[d]);
      atomicAdd(vi + 3 * ib + d, imp[d]);
    }
  }
}

// advance_toi (solver_mass_spring.py:117-148) in place; consumes v_inc and
// leaves it zero for the next substep
__global__ void na_advance(cls_noalloc_advance a, float drag_s, float* __restrict__ vinc) {
  const long long total = (long long)a.n_envs * a.n_vertices;
  cls::MsArgs<float> p;
  p.dt = a.dt;
  p.gravity = a.gravity;
  p.ground = a.ground_height;
  p.drag_s = drag_s;
  p.friction = a.friction;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
       q += (long long)gridDim.x * blockDim.x) {
    float* xq = a.x + 3 * q;
    float* vq = a.v + 3 * q;
    float* iq = vinc + 3 * q;
    cls::V4<float> x, v, vi;
    x.x = xq[0]; x.y = xq[1]; x.z = xq[2]; x.w = 0;
    v.x = vq[0]; v.y = vq[1]; v.z = vq[2]; v.w = 0;
    vi.x = iq[0]; vi.y = iq[1]; vi.z = iq[2]; vi.w = 0;
    cls::advance_vertex<float>(p, x, v, vi);
    xq[0] = x.x; xq[1] = x.y; xq[2] = x.z;
    vq[0] = v.x; vq[1] = v.y; vq[2] = v.z;
    iq[0] = 0.f; iq[1] = 0.f; iq[2] = 0.f;
  }
}

// All substeps of one env in one CTA: positions, velocities, spring constants and
// impulses stay in shared memory, so a call is one launch instead of two per
// substep.  The springs' impulses are evaluated spring-parallel into a table and
// summed per vertex in spring order (a row list built at the start), without
// atomics.  Bound by the latency of its three barriers per substep and of the
// impulse's arithmetic: 64 quadrupeds (93 vertices, 608 springs) 10.3 -> 1.9 us per
// substep (two launches and six global atomics per spring before).
struct FusedShared {
  cls::V4<float>* x;
  cls::V4<float>* v;
  cls::V4<float>* imp;     // per spring
  float4* par;             // per spring: rest length, stiffness, coefficient, actuation
  ushort2* ab;             // per spring: endpoints (both kNone: skipped)
  unsigned short* inc;     // per vertex, in spring order: 2 spring + side
  int* ptr;                // n_vertices + 1 row starts
};
constexpr unsigned short kNone = 0xffff;
constexpr int kFusedMax = 32767;   // springs (2 s + side in 16 bits) and vertices
// incidences of a vertex that one thread sorts and sums, twice the cube lattices'
// largest degree; beyond it a warp takes the vertex (900 vertices, 4600 springs, one
// with 900 of them, one substep: 2830 us when its thread sorted and summed them
// alone, 44 now)
constexpr int kThreadRow = 48;
constexpr int kFillMax = 12;       // incidences per thread while the rows are sorted

__host__ __device__ inline size_t carve_fused(char* base, int nv, int ns, FusedShared* s) {
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += (bytes + 15) & ~size_t(15); return p; };
  FusedShared z;
  z.x = (cls::V4<float>*)take(sizeof(cls::V4<float>) * nv);
  z.v = (cls::V4<float>*)take(sizeof(cls::V4<float>) * nv);
  z.imp = (cls::V4<float>*)take(sizeof(cls::V4<float>) * ns);
  z.par = (float4*)take(sizeof(float4) * ns);
  z.ab = (ushort2*)take(sizeof(ushort2) * ns);
  z.inc = (unsigned short*)take(sizeof(unsigned short) * 2 * ns);
  z.ptr = (int*)take(sizeof(int) * (nv + 1));
  if (s) *s = z;
  return off;
}

// work(h), by a whole warp, for every vertex h whose row is longer than one thread
// takes; the warps take every nw-th vertex, so that neighbouring hubs are shared out
template <typename Work>
__device__ __forceinline__ void na_hubs(const FusedShared& s, int N, Work work) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i0 = wid; i0 < N; i0 += 32 * nw) {
    const int i = i0 + nw * lane;
    unsigned rows = __ballot_sync(0xffffffffu, i < N && s.ptr[i < N ? i + 1 : 0] - s.ptr[i < N ? i : 0] > kThreadRow);
    for (; rows; rows &= rows - 1) work(i0 + nw * (__ffs(rows) - 1));
  }
}

// The thread's springs tid, tid + blockDim, ..: their ends, all loads in flight at once
// (-1, -1 beyond the last and where an end is outside the robot).
constexpr int kSpringMax = kFillMax / 2;   // per thread
__device__ __forceinline__ void na_ends(const cls_noalloc_advance& a, int2 (&ab)[kSpringMax]) {
  const int S = a.n_springs, N = a.n_vertices;
#pragma unroll
  for (int k = 0; k < kSpringMax; ++k) {
    const int q = threadIdx.x + k * blockDim.x;
    ab[k] = q < S ? make_int2(a.spring_a[q], a.spring_b[q]) : make_int2(-1, -1);
  }
#pragma unroll
  for (int k = 0; k < kSpringMax; ++k)
    if (ab[k].x < 0 || ab[k].x >= N || ab[k].y < 0 || ab[k].y >= N) ab[k] = make_int2(-1, -1);
}

// counts ptr[1 .. n] to row starts ptr[0 .. n] (ptr[0] = 0), by all threads; part: n / 32 + 1
// ints.  Ends with a barrier.
__device__ __forceinline__ void na_row_starts(int* ptr, int n, int* part) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto scan = [&](int c) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) c += up;
    }
    return c;
  };
  __syncthreads();
  for (int g = wid; 32 * g <= n; g += nw) {
    const int i = 32 * g + lane, c = scan(i <= n ? ptr[i] : 0);
    if (i <= n) ptr[i] = c;
    if (lane == 31) part[g] = c;
  }
  __syncthreads();
  if (wid == 0) {
    int carry = 0;
    for (int g0 = 0; 32 * g0 <= n; g0 += 32) {
      const int g = g0 + lane, c = carry + scan(32 * g <= n ? part[g] : 0);
      if (32 * g <= n) part[g] = c;
      carry = __shfl_sync(0xffffffffu, c, 31);
    }
  }
  __syncthreads();
  for (int i = 32 + threadIdx.x; i <= n; i += blockDim.x) ptr[i] += part[(i >> 5) - 1];
  __syncthreads();
}

__global__ void __launch_bounds__(1024) na_fused(cls_noalloc_advance a, float drag_s) {
  extern __shared__ __align__(16) char na_smem[];
  FusedShared s;
  carve_fused(na_smem, a.n_vertices, a.n_springs, &s);
  const int tid = threadIdx.x, nt = blockDim.x, N = a.n_vertices, S = a.n_springs;
  float* xe = a.x + (size_t)blockIdx.x * N * 3;
  float* ve = a.v + (size_t)blockIdx.x * N * 3;
  for (int i = tid; i < N; i += nt) {
    cls::V4<float> x, v;
    x.x = xe[3 * i]; x.y = xe[3 * i + 1]; x.z = xe[3 * i + 2]; x.w = 0;
    v.x = ve[3 * i]; v.y = ve[3 * i + 1]; v.z = ve[3 * i + 2]; v.w = 0;
    s.x[i] = x;
    s.v[i] = v;
  }
  for (int i = tid; i <= N; i += nt) s.ptr[i] = 0;
  int2 ab[kSpringMax];
  na_ends(a, ab);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kSpringMax; ++k) {
    const int q = tid + k * nt;
    if (q < S) s.ab[q] = make_ushort2((unsigned short)ab[k].x, (unsigned short)ab[k].y);  // -1: kNone
    if (ab[k].x < 0) continue;
    atomicAdd(s.ptr + ab[k].x + 1, 1);
    atomicAdd(s.ptr + ab[k].y + 1, 1);
  }
#pragma unroll
  for (int k = 0; k < kSpringMax; ++k) {
    const int q = tid + k * nt;
    if (q < S)
      s.par[q] = make_float4(a.rest_length[q], a.stiffness[q], a.actuation_coef[q], a.actuation[(size_t)blockIdx.x * S + q]);
  }
  int* fill = reinterpret_cast<int*>(s.v);   // the velocities come back below
  na_row_starts(s.ptr, N, fill);
  // rows in any order, then sorted; the long rows of hub vertices are written in
  // order by a warp each (na_hubs)
  bool long_row = false;
  for (int i = tid; i < N; i += nt) long_row |= s.ptr[i + 1] - s.ptr[i] > kThreadRow;
  const bool hubs = __syncthreads_or(long_row);
  for (int i = tid; i < N; i += nt) fill[i] = s.ptr[i];
  __syncthreads();
  auto by_thread = [&](int i) { return !hubs || s.ptr[i + 1] - s.ptr[i] <= kThreadRow; };
#pragma unroll
  for (int k = 0; k < kSpringMax; ++k) {
    if (ab[k].x < 0) continue;
    const int q = tid + k * nt;
    if (by_thread(ab[k].x)) s.inc[atomicAdd(fill + ab[k].x, 1)] = (unsigned short)(2 * q);
    if (by_thread(ab[k].y)) s.inc[atomicAdd(fill + ab[k].y, 1)] = (unsigned short)(2 * q + 1);
  }
  const int lane = tid & 31;
  const unsigned below = (1u << lane) - 1u;
  if (hubs)
    na_hubs(s, N, [&](int h) {
      int at = s.ptr[h];
      for (int q0 = 0; q0 < S; q0 += 32) {
        const int q = q0 + lane;
        const ushort2 ab = q < S ? s.ab[q] : make_ushort2(kNone, kNone);
        const unsigned in_a = __ballot_sync(0xffffffffu, ab.x == h), in_b = __ballot_sync(0xffffffffu, ab.y == h);
        int p = at + __popc(in_a & below) + __popc(in_b & below);
        if (ab.x == h) s.inc[p++] = (unsigned short)(2 * q);
        if (ab.y == h) s.inc[p] = (unsigned short)(2 * q + 1);
        at += __popc(in_a) + __popc(in_b);
      }
    });
  __syncthreads();
  // a thread per incidence: its place in its row is the number of smaller ones (one
  // quadruped, 608 springs, one substep: 10.4 us a call, 18.7 with a row sorted by its
  // vertex's thread)
  {
    unsigned short code[kFillMax];
    int to[kFillMax];
    const int n_inc = s.ptr[N];
#pragma unroll
    for (int k = 0; k < kFillMax; ++k) {
      const int at = tid + k * nt;
      to[k] = -1;
      if (at >= n_inc) continue;
      code[k] = s.inc[at];
      const ushort2 ab = s.ab[code[k] >> 1];
      const int i = (code[k] & 1) ? ab.y : ab.x;
      const int b = s.ptr[i], e = s.ptr[i + 1];
      if (e - b > kThreadRow) continue;
      int rank = 0;
#pragma unroll 8
      for (int p = b; p < e; ++p) rank += s.inc[p] < code[k];
      to[k] = b + rank;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFillMax; ++k)
      if (to[k] >= 0) s.inc[to[k]] = code[k];
  }
  for (int i = tid; i < N; i += nt) {
    cls::V4<float> v;
    v.x = ve[3 * i]; v.y = ve[3 * i + 1]; v.z = ve[3 * i + 2]; v.w = 0;
    s.v[i] = v;
  }
  cls::MsArgs<float> p;
  p.dt = a.dt;
  p.gravity = a.gravity;
  p.ground = a.ground_height;
  p.drag_s = drag_s;
  p.friction = a.friction;
  __syncthreads();
  for (int step = 0; step < a.n_substeps; ++step) {
    for (int q = tid; q < S; q += nt) {
      const ushort2 ab = s.ab[q];
      if (ab.x == kNone) continue;
      const float4 c = s.par[q];
      float imp[3];
      cls::spring_impulse<float>(s.x[ab.x], s.x[ab.y], s.v[ab.x], s.v[ab.y], c.x, c.y, c.z, c.w, a.dt,
                                 a.dashpot_damping, imp);
      cls::V4<float> r;
      r.x = imp[0]; r.y = imp[1]; r.z = imp[2]; r.w = 0;
      s.imp[q] = r;
    }
    __syncthreads();
    for (int i = tid; i < N; i += nt) {
      cls::V4<float> vi;
      vi.x = vi.y = vi.z = vi.w = 0;
      const int e = s.ptr[i + 1];
      if (e - s.ptr[i] > kThreadRow) continue;
#pragma unroll 4
      for (int k = s.ptr[i]; k < e; ++k) {
        const int c = s.inc[k];
        const cls::V4<float> r = s.imp[c >> 1];
        if (c & 1) { vi.x += r.x; vi.y += r.y; vi.z += r.z; }
        else { vi.x -= r.x; vi.y -= r.y; vi.z -= r.z; }
      }
      cls::V4<float> x = s.x[i], v = s.v[i];
      cls::advance_vertex<float>(p, x, v, vi);
      s.x[i] = x;
      s.v[i] = v;
    }
    if (hubs)
      na_hubs(s, N, [&](int h) {
        cls::V4<float> vi;
        vi.x = vi.y = vi.z = vi.w = 0;
        for (int k = s.ptr[h] + lane; k < s.ptr[h + 1]; k += 32) {
          const int c = s.inc[k];
          const cls::V4<float> r = s.imp[c >> 1];
          if (c & 1) { vi.x += r.x; vi.y += r.y; vi.z += r.z; }
          else { vi.x -= r.x; vi.y -= r.y; vi.z -= r.z; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          vi.x += __shfl_xor_sync(0xffffffffu, vi.x, o);
          vi.y += __shfl_xor_sync(0xffffffffu, vi.y, o);
          vi.z += __shfl_xor_sync(0xffffffffu, vi.z, o);
        }
        if (lane == 0) {
          cls::V4<float> x = s.x[h], v = s.v[h];
          cls::advance_vertex<float>(p, x, v, vi);
          s.x[h] = x;
          s.v[h] = v;
        }
      });
    __syncthreads();
  }
  for (int i = tid; i < N; i += nt) {
    const cls::V4<float> x = s.x[i], v = s.v[i];
    xe[3 * i] = x.x; xe[3 * i + 1] = x.y; xe[3 * i + 2] = x.z;
    ve[3 * i] = v.x; ve[3 * i + 1] = v.y; ve[3 * i + 2] = v.z;
  }
}

// The same with a cluster of C CTAs per env, for calls of few envs: each CTA holds the
// positions and velocities of the whole env, and the lists, impulses and sums of its own
// vertices -- an incidence's impulse is evaluated for its own vertex, a thread per
// incidence, and summed in na_fused's order.  Every substep ends with the new state
// stored into all CTAs of the cluster.  What one CTA of na_fused takes one after another
// for thousands of springs (900 vertices, 4600 springs: 23 us for a call of one substep, 244
// of 32) is C times less here (13.4 and 128 with C = 8).  Bound by the latency of a call's
// dozen short phases.
constexpr int kSliceHeld = 2;      // incidences of a thread whose springs stay in registers

struct SliceShared {
  cls::V4<float>* x;
  cls::V4<float>* v;
  cls::V4<float>* imp;     // per own incidence, the first slice_table(..) of them
  cls::V4<float>* sum;     // per own vertex
  unsigned short* inc;     // per own vertex in spring order: 2 spring + side (room for all)
  int* ptr;                // row starts of the own vertices, + 1
  int* fill;
};
// Twice the balanced share: with room for every incidence, which one CTA could own,
// little L1 is left (4600 springs, one substep, C = 8: 16.7 us).  Those beyond the table
// are evaluated as their row is summed.
__host__ __device__ inline int slice_table(int ns, int C) { return 4 * ns / C + 32; }

__host__ __device__ inline size_t carve_slices(char* base, int nv, int ns, int C, SliceShared* s) {
  size_t off = 0;
  auto take = [&](size_t bytes) { char* p = base + off; off += (bytes + 15) & ~size_t(15); return p; };
  SliceShared z;
  z.x = (cls::V4<float>*)take(sizeof(cls::V4<float>) * nv);
  z.v = (cls::V4<float>*)take(sizeof(cls::V4<float>) * nv);
  z.imp = (cls::V4<float>*)take(sizeof(cls::V4<float>) * slice_table(ns, C));
  z.sum = (cls::V4<float>*)take(sizeof(cls::V4<float>) * (nv / C + 1));
  z.inc = (unsigned short*)take(sizeof(unsigned short) * 2 * ns);
  z.ptr = (int*)take(sizeof(int) * (nv + 1));
  z.fill = (int*)take(sizeof(int) * nv);
  if (s) *s = z;
  return off;
}

__global__ void __launch_bounds__(1024) na_slices(cls_noalloc_advance a, float drag_s) {
  extern __shared__ __align__(16) char na_smem[];
  const int C = (int)cls::cl::size();
  SliceShared s;
  carve_slices(na_smem, a.n_vertices, a.n_springs, C, &s);
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, N = a.n_vertices, S = a.n_springs;
  const int cap = slice_table(S, C), rank = (int)cls::cl::rank(), env = (int)blockIdx.x / C;
  const int v0 = (int)((long long)N * rank / C), M = (int)((long long)N * (rank + 1) / C) - v0;
  float* xe = a.x + (size_t)env * N * 3;
  float* ve = a.v + (size_t)env * N * 3;
  const float* act = a.actuation + (size_t)env * S;
  for (int i = tid; i < N; i += nt) {
    cls::V4<float> x, v;
    x.x = xe[3 * i]; x.y = xe[3 * i + 1]; x.z = xe[3 * i + 2]; x.w = 0;
    v.x = ve[3 * i]; v.y = ve[3 * i + 1]; v.z = ve[3 * i + 2]; v.w = 0;
    s.x[i] = x;
    s.v[i] = v;
  }
  for (int i = tid; i <= M; i += nt) s.ptr[i] = 0;
  int2 ab[kSpringMax];
  na_ends(a, ab);
  // own(f): f(own vertex, 2 spring + side) for the own ends of the thread's springs
  auto own = [&](auto f) {
#pragma unroll
    for (int k = 0; k < kSpringMax; ++k) {
      const int q = tid + k * nt;
      if (ab[k].x < 0) continue;
      if (ab[k].x >= v0 && ab[k].x < v0 + M) f(ab[k].x - v0, 2 * q);
      if (ab[k].y >= v0 && ab[k].y < v0 + M) f(ab[k].y - v0, 2 * q + 1);
    }
  };
  __syncthreads();
  own([&](int i, int) { atomicAdd(s.ptr + i + 1, 1); });
  na_row_starts(s.ptr, M, s.fill);
  bool long_row = false;
  for (int i = tid; i < M; i += nt) {
    s.fill[i] = s.ptr[i];
    long_row |= s.ptr[i + 1] - s.ptr[i] > kThreadRow;
  }
  const bool hubs = __syncthreads_or(long_row);
  own([&](int i, int code) { s.inc[atomicAdd(s.fill + i, 1)] = (unsigned short)code; });
  __syncthreads();
  const int n_inc = s.ptr[M];
  {  // a thread per incidence: its place in its row is the number of smaller ones
    unsigned short code[kFillMax];
    int to[kFillMax];
#pragma unroll
    for (int k = 0; k < kFillMax; ++k) {
      const int at = tid + k * nt;
      to[k] = -1;
      if (at >= n_inc) continue;
      code[k] = s.inc[at];
      const int i = ((code[k] & 1) ? a.spring_b : a.spring_a)[code[k] >> 1] - v0;
      int r = s.ptr[i];
      for (int p = s.ptr[i], e = s.ptr[i + 1]; p < e; ++p) r += s.inc[p] < code[k];
      to[k] = r;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFillMax; ++k)
      if (to[k] >= 0) s.inc[to[k]] = code[k];
  }
  cls::MsArgs<float> p;
  p.dt = a.dt;
  p.gravity = a.gravity;
  p.ground = a.ground_height;
  p.drag_s = drag_s;
  p.friction = a.friction;
  __syncthreads();
  // the springs of the thread's incidences; the first ones stay in registers
  struct Spring {
    int a, b;
    float4 c;
  };
  auto spring = [&](int k) {
    const int q = s.inc[k] >> 1;
    Spring g;
    g.a = a.spring_a[q];
    g.b = a.spring_b[q];
    g.c = make_float4(a.rest_length[q], a.stiffness[q], a.actuation_coef[q], act[q]);
    return g;
  };
  auto impulse = [&](const Spring& g) {
    float imp[3];
    cls::spring_impulse<float>(s.x[g.a], s.x[g.b], s.v[g.a], s.v[g.b], g.c.x, g.c.y, g.c.z, g.c.w, a.dt,
                               a.dashpot_damping, imp);
    cls::V4<float> r;
    r.x = imp[0]; r.y = imp[1]; r.z = imp[2]; r.w = 0;
    return r;
  };
  const int n_tab = n_inc < cap ? n_inc : cap;
  Spring held[kSliceHeld];
#pragma unroll
  for (int k = 0; k < kSliceHeld; ++k)
    if (tid + k * nt < n_tab) held[k] = spring(tid + k * nt);
  for (int step = 0; step < a.n_substeps; ++step) {
#pragma unroll
    for (int k = 0; k < kSliceHeld; ++k)
      if (tid + k * nt < n_tab) s.imp[tid + k * nt] = impulse(held[k]);
    for (int k = tid + kSliceHeld * nt; k < n_tab; k += nt) s.imp[k] = impulse(spring(k));
    __syncthreads();
    auto add = [&](int k, cls::V4<float>& vi) {
      const cls::V4<float> r = k < cap ? s.imp[k] : impulse(spring(k));
      if (s.inc[k] & 1) { vi.x += r.x; vi.y += r.y; vi.z += r.z; }
      else { vi.x -= r.x; vi.y -= r.y; vi.z -= r.z; }
    };
    for (int i = tid; i < M; i += nt) {
      cls::V4<float> vi;
      vi.x = vi.y = vi.z = vi.w = 0;
      const int e = s.ptr[i + 1];
      if (e - s.ptr[i] > kThreadRow) continue;
#pragma unroll 4
      for (int k = s.ptr[i]; k < e; ++k) add(k, vi);
      s.sum[i] = vi;
    }
    if (hubs) {
      FusedShared rows;
      rows.ptr = s.ptr;
      na_hubs(rows, M, [&](int h) {
        cls::V4<float> vi;
        vi.x = vi.y = vi.z = vi.w = 0;
        for (int k = s.ptr[h] + lane; k < s.ptr[h + 1]; k += 32) add(k, vi);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          vi.x += __shfl_xor_sync(0xffffffffu, vi.x, o);
          vi.y += __shfl_xor_sync(0xffffffffu, vi.y, o);
          vi.z += __shfl_xor_sync(0xffffffffu, vi.z, o);
        }
        if (lane == 0) s.sum[h] = vi;
      });
    }
    // all CTAs have read the state (before the first substep: the caller's arrays too)
    cls::cl::sync();
    for (int i = tid; i < M; i += nt) {
      cls::V4<float> x = s.x[v0 + i], v = s.v[v0 + i];
      cls::advance_vertex<float>(p, x, v, s.sum[i]);
      if (step + 1 < a.n_substeps) {
        for (int r = 0; r < C; ++r) {
          *cls::cl::peer(s.x + v0 + i, r) = x;
          *cls::cl::peer(s.v + v0 + i, r) = v;
        }
      } else {
        const int g = 3 * (v0 + i);
        xe[g] = x.x; xe[g + 1] = x.y; xe[g + 2] = x.z;
        ve[g] = v.x; ve[g + 1] = v.y; ve[g + 2] = v.z;
      }
    }
    if (step + 1 < a.n_substeps) cls::cl::sync();
  }
}

// largest dynamic shared memory of na_fused on the current device (0: unknown) and
// its SMs
size_t fused_capacity(int* n_sm) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return (size_t)optin;
}

// Threads of na_fused.  With more envs than SMs, 512 where two CTAs' shared memory fits
// an SM, whose threads two of 1024 would fill (600 spiders, one / 32 substeps: 49 / 474 ->
// 35 / 372 us).
int fused_threads(const cls_noalloc_advance& a, int n_sm, size_t smem, size_t most) {
  const int work = a.n_springs > a.n_vertices ? a.n_springs : a.n_vertices;
  const bool pairs = a.n_envs > n_sm && work <= kSpringMax * 512 && 2 * smem <= most;
  return work <= 256 ? 256 : (work <= 1024 || pairs ? 512 : 1024);
}

// CTAs per env of na_slices, 1 for na_fused: clusters that can all run at once (8 up to
// 12 envs, 4 up to 29 on 148 SMs), from where they are the faster form for calls of any
// length (na_fused / na_slices, us, one env, 1 and 32 substeps: 1000 springs 10.5 / 10.5 and
// 80 / 85, 1378 12.5 / 10.5 and 98 / 94, 3000 16.8 / 12.5 and 164 / 107, 4600 22.8 / 13.4 and
// 242 / 128; 29 envs of 1378 12.5 / 11.3 and 99 / 99).
constexpr int kSliceSprings = 1300, kSliceThreads = 1024;
int slice_count(const cls_noalloc_advance& a, int n_sm) {
  if (a.n_springs < kSliceSprings || 2 * a.n_springs > kFillMax * kSliceThreads) return 1;
  return 12LL * a.n_envs <= n_sm ? 8 : (5LL * a.n_envs <= n_sm ? 4 : 1);
}

int grid_for(long long n) {
  long long g = (n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  return g < 1 ? 1 : (int)g;
}

}  // namespace

extern "C" int cls_ms_advance_noalloc(const cls_noalloc_advance* a, void* stream) {
  if (!a) return CLS_ERR_INVALID;
  if (a->n_envs <= 0 || a->n_vertices <= 0 || a->n_springs < 0 || a->n_substeps < 0 || !a->x ||
      !a->v || (a->n_springs > 0 && (!a->spring_a || !a->spring_b || !a->rest_length ||
                                     !a->stiffness || !a->actuation_coef || !a->actuation))) {
    set_message(a, "cls_ms_advance_noalloc: missing pointer or non-positive size");
    return CLS_ERR_INVALID;
  }
  const long long need = (long long)a->n_envs * a->n_vertices * 3;
  if (need > kScratchFloats) {
    char msg[200];
    snprintf(msg, sizeof(msg),
             "cls_ms_advance_noalloc: n_envs * n_vertices * 3 = %lld exceeds the fixed scratch of "
             "%lld floats",
             need, kScratchFloats);
    set_message(a, msg);
    return CLS_ERR_INVALID;
  }
  // an error left by the caller's earlier work stays pending for the caller
  const cudaError_t pending = cudaPeekAtLastError();
  if (pending != cudaSuccess) {
    char msg[200];
    snprintf(msg, sizeof(msg),
             "cls_ms_advance_noalloc: a CUDA error from earlier work is pending (%s); nothing "
             "launched",
             cudaGetErrorName(pending));
    set_message(a, msg);
    return CLS_ERR_CUDA;
  }
  float* scratch = nullptr;
  const cudaError_t se = scratch_address(&scratch);
  if (se != cudaSuccess) {
    set_message(a, cudaGetErrorString(se));
    return CLS_ERR_CUDA;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const float drag_s = (float)exp(-(double)a->dt * (double)a->drag_damping);
  // one CTA (or cluster) per env when an env's springs fit in a CTA's shared memory (up to
  // about 5000 springs); larger ones keep a launch per phase over the scratch array
  const size_t smem = carve_fused(nullptr, a->n_vertices, a->n_springs, nullptr);
  int n_sm = 0;
  const size_t fused_max = fused_capacity(&n_sm);
  const int threads = fused_threads(*a, n_sm, smem, fused_max);
  if (a->n_substeps > 0 && a->n_vertices <= kFusedMax && 2 * a->n_springs <= kFillMax * threads &&
      smem <= fused_max) {
    // the limit belongs to the kernel in the whole process: always the device's
    // maximum, so that a call with a smaller robot on another host thread never
    // lowers it between this call's raise and its launch
    const int slices = slice_count(*a, n_sm);
    const size_t bytes = carve_slices(nullptr, a->n_vertices, a->n_springs, slices, nullptr);
    if (slices > 1 && bytes <= fused_max) {
      cudaError_t e = cudaFuncSetAttribute(na_slices, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_max);
      cudaLaunchConfig_t c{};
      cudaLaunchAttribute at{};
      c.gridDim = dim3((unsigned)(a->n_envs * slices));
      c.blockDim = dim3(kSliceThreads);
      c.dynamicSmemBytes = bytes;
      c.stream = s;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = (unsigned)slices;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      c.attrs = &at;
      c.numAttrs = 1;
      if (e == cudaSuccess) e = cudaLaunchKernelEx(&c, na_slices, *a, drag_s);
      if (e == cudaSuccess) return CLS_OK;
      cudaGetLastError();  // a device that cannot hold such a cluster: one CTA
    }
    cudaError_t e = smem > 48 * 1024
                        ? cudaFuncSetAttribute(na_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_max)
                        : cudaSuccess;
    if (e == cudaSuccess) {
      na_fused<<<a->n_envs, threads, smem, s>>>(*a, drag_s);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
      cudaGetLastError();  // this call's own error: reported here, not left for the next call
      set_message(a, cudaGetErrorString(e));
      return CLS_ERR_CUDA;
    }
    return CLS_OK;
  }
  na_clear<<<grid_for(need), 256, 0, s>>>(scratch, need);
  for (int step = 0; step < a->n_substeps; ++step) {
    if (a->n_springs > 0)
      na_spring<<<grid_for((long long)a->n_envs * a->n_springs), 256, 0, s>>>(*a, scratch);
    na_advance<<<grid_for((long long)a->n_envs * a->n_vertices), 256, 0, s>>>(*a, drag_s, scratch);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_message(a, cudaGetErrorString(e));
    return CLS_ERR_CUDA;
  }
  return CLS_OK;
}
