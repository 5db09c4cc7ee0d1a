// mpm_small.cu -- the one-CTA-per-env MPM rollouts (mpm_small.cuh) in their own
// module.
#include "mpm_small.cuh"

namespace cls {
namespace mpm {

namespace {
long long node_count(int D, int n_grid) {
  long long n = 1;
  for (int d = 0; d < D; ++d) n *= n_grid;
  return n;
}
template <typename R, int D>
size_t fwd_bytes(int P, int n_grid, int cap) {
  return carve<R, D>(nullptr, P, (int)node_count(D, n_grid), cap, (SmallFwdShared<R, D>*)nullptr);
}
template <typename R, int D>
size_t adj_bytes(int P, int n_grid, int cap) {
  return carve<R, D>(nullptr, P, (int)node_count(D, n_grid), cap, (SmallAdjShared<R, D>*)nullptr);
}
template <typename R>
__global__ void seed_kernel(SeedChunk<R> c) {
  for (int i = threadIdx.x; i < c.n; i += blockDim.x) c.out[i] = c.w[i];
}

// one warp per 32 particles, enough threads for the grid phase
int threads(int P) {
  const int t = (P + 31) / 32 * 32;
  return t < 256 ? 256 : (t > kSmallThreads ? kSmallThreads : t);
}
}  // namespace

template <typename R, int D>
cudaError_t SmallLaunch<R, D>::plan(int E, int P, int n_grid, bool* ok, int* fwd_cap, int* adj_cap) {
  *ok = false;
  if (n_grid < 3 || n_grid > 1000 || node_count(D, n_grid) > (1 << 15)) return cudaSuccess;
  int dev = 0, optin = 0, n_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess || !small_body(D, E, P, n_sm)) return e;
  // a run per particle at most; smaller tables where that does not fit, down to
  // one per four particles (the voxelised bodies' runs), else the general kernels
  int caps[2] = {0, 0};
  for (int k = 0; k < 2; ++k) {
    auto fits = [&](int cap) {
      return (k ? adj_bytes<R, D>(P, n_grid, cap) : fwd_bytes<R, D>(P, n_grid, cap)) <= (size_t)optin;
    };
    int lo = (P + 3) / 4, hi = P;
    if (!fits(lo)) return cudaSuccess;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (fits(mid)) lo = mid; else hi = mid - 1;
    }
    caps[k] = lo;
  }
  // the device's maximum: handles of different sizes share the attribute
  e = cudaFuncSetAttribute(mpm_small_fwd_kernel<R, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(mpm_small_adj_kernel<R, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  // more envs than SMs: only where an SM holds two
  int nf = 2, nr = 2;
  if (E > n_sm) {
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nf, mpm_small_fwd_kernel<R, D>, threads(P),
                                                        fwd_bytes<R, D>(P, n_grid, caps[0]));
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nr, mpm_small_adj_kernel<R, D>, threads(P),
                                                        adj_bytes<R, D>(P, n_grid, caps[1]));
  }
  *ok = e == cudaSuccess && nf >= 2 && nr >= 2;
  *fwd_cap = caps[0];
  *adj_cap = caps[1];
  return e;
}

template <typename R, int D>
cudaError_t SmallLaunch<R, D>::forward(const SmallFwdArgs<R>& a, cudaStream_t s) {
  mpm_small_fwd_kernel<R, D><<<a.c.E, threads(a.c.P), fwd_bytes<R, D>(a.c.P, a.c.n_grid, a.cap), s>>>(a);
  return cudaGetLastError();
}
template <typename R, int D>
cudaError_t SmallLaunch<R, D>::reverse(const SmallAdjArgs<R>& a, cudaStream_t s) {
  mpm_small_adj_kernel<R, D><<<a.c.E, threads(a.c.P), adj_bytes<R, D>(a.c.P, a.c.n_grid, a.cap), s>>>(a);
  return cudaGetLastError();
}

template <typename R, int D>
cudaError_t SmallLaunch<R, D>::seeds(const double* w, int n, R* out, cudaStream_t s) {
  SeedChunk<R> c;
  for (int i0 = 0; i0 < n; i0 += c.kMax) {
    c.n = n - i0 < c.kMax ? n - i0 : c.kMax;
    c.out = out + i0;
    for (int i = 0; i < c.n; ++i) c.w[i] = (R)w[i0 + i];
    seed_kernel<R><<<1, 256, 0, s>>>(c);
  }
  return cudaGetLastError();
}

template struct SmallLaunch<float, 2>;
template struct SmallLaunch<float, 3>;
template struct SmallLaunch<double, 2>;
template struct SmallLaunch<double, 3>;

}  // namespace mpm
}  // namespace cls
