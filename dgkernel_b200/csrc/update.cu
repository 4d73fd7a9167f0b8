// Elementwise update kernels (updateSolution, lserkUpdate).
#include <algorithm>
#include <cstdint>

#include "dg_kernels.cuh"
#include "launch.cuh"

namespace dgk {

// Elementwise updates over runs of kUpdateValues values: mode 0 = the reference's updateSolution
// (resu = rka*resu + rkb*rhsu; u += resu), mode 1 = standard LSERK4 (resu = a*resu + dt*rhs; u += b*resu).
// Bound by HBM: a run is four loads of each array per thread, all in flight, and a block of its own, so that every block
// has a full run whatever the values per element (16 M values: FP64 94 us, 6.8 TB/s; FP32 49).  Tiles of 64 elements held
// a quarter of those loads at 4 values per element (FP64 154 us, FP32 136) and ragged tails at others (35: 111 and 68);
// runs walked by a grid of eight blocks an SM took 106 and 54.  Launched behind the kernel that forms the right-hand side
// (pdl_wait), with the run's place already read: order 1, 48^3 x 6 FP64, computeRHS and update 56.2 -> 53.5 us.
template <typename T>
__global__ void __launch_bounds__(kUpdateThreads) update_kernel(const Tile *runs, int nruns, T *u, T *resu, const T *rhs,
                                                                T c0, T c1, T c2, int mode) {
  constexpr int CH = kUpdateValues / kUpdateThreads;
  for (int t = blockIdx.x; t < nruns; t += gridDim.x) {
    const Tile run = runs[t];
    pdl_wait();
    const int n = run.nelem;
    T *pr = resu + run.node_base, *pu = u + run.node_base;
    const T *pw = rhs + run.node_base;
    T r[CH], v[CH], w[CH];
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int x = threadIdx.x + j * kUpdateThreads;
      r[j] = x < n ? pr[x] : T(0);
      v[j] = x < n ? pu[x] : T(0);
      w[j] = x < n ? pw[x] : T(0);
    }
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int x = threadIdx.x + j * kUpdateThreads;
      if (x < n) {
        const T res = mode == 0 ? c0 * r[j] + c1 * w[j] : c0 * r[j] + c2 * w[j];
        pr[x] = res;
        pu[x] = mode == 0 ? v[j] + res : v[j] + c1 * res;
      }
    }
  }
}

template <typename T>
void launch_update(const Tile *runs, int nruns, T *u, T *resu, const T *rhs, double c0, double c1, double c2, int mode,
                   cudaStream_t st) {
  const int grid = std::min(nruns, 1 << 20);
  if (grid > 0)
    launch_pdl(update_kernel<T>, grid, kUpdateThreads, 0, st, runs, nruns, u, resu, rhs, (T)c0, (T)c1, (T)c2, mode);
}

template void launch_update<double>(const Tile *, int, double *, double *, const double *, double, double, double, int,
                                    cudaStream_t);
template void launch_update<float>(const Tile *, int, float *, float *, const float *, double, double, double, int,
                                    cudaStream_t);

}  // namespace dgk
