// Fused strong-form Lax-Friedrichs RHS + LSERK4 stage at orders 6 and 7, arrays in FP64 or FP32 (T), where the reference
// matrices (237 and 483 KB) fit neither registers nor shared memory.
//
// The products run on the FP64 tensor path (mma.sync m8n8k4) with the matrices streamed from L2: the operator stores
// them in fragment order, so a warp's A fragment is 256 consecutive bytes, loaded two k-steps ahead and used for NT
// n-tiles of 8 elements.  A CTA holds one tile of 8 NT elements: state, volume terms and face terms in shared memory
// (51 KB at order 7 and NT = 2), rows stored at strides of 4 or 12 mod 16 values, which keeps the fragment loads free
// of bank conflicts.  The nine metrics and four face arrays are read once, straight from global memory, 64 consecutive
// bytes per element.  They are brought into L2 by bulk prefetches shortly before their phase: prefetched a whole tile
// ahead, the CTAs' tiles together outgrow L2, and prefetched ahead of a phase that loads itself, they delay it (order 7,
// 16^3 x 6, measured on tiles of 32 elements, a shape since removed: 1012 us per LSERK4 step a tile ahead, 860 as here).
// Several small CTAs share an SM and drift apart, so one's memory phases run under another's products: three CTAs of 16
// elements take 775 us, two of 16 take 840 and two of 32 take 860.  Each warp owns one or two 8-row m-tiles.
//
// Bound by the FP64 rate (60,480 FMAs per element at order 7, 82 us of the 155 us per stage) and by the latency of
// the memory phases.  The form before it read a matrix entry per FMA through L1: 655 us per stage.
#include <algorithm>
#include <cstdint>

#include "dg_kernels.cuh"
#include "launch.cuh"

namespace dgk {

namespace {

template <int N, int NT>
struct WideCfg {
  using O = Order<N>;
  static constexpr int NP = O::NP, NF = O::NF;
  static constexpr int TE = 8 * NT;
  static constexpr int MT = (NP + 7) / 8, KT = NP / 4, KL = NF / 4;
  static constexpr int WARPS = (MT + 1) / 2;  // one or two m-tiles per warp
  static constexpr int THREADS = 32 * WARPS;
  static constexpr int MINB = N == 6 ? 4 : 3;  // CTAs per SM
  static constexpr int SU = frag_stride(NP), SF = frag_stride(NF);
  static constexpr size_t SMEM = sizeof(double) * (size_t)TE * (2 * SU + SF) + sizeof(int) * NF;
  static constexpr int DEPTH = 3;  // A fragments in flight
  static_assert(NP % 4 == 0 && NF % 16 == 0 && KT % DEPTH == 0, "whole k-steps");
};

__device__ __forceinline__ void wide_dmma(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// A matrix fragment's load, kept where it is written: as a plain load the compiler moves it down to its use
__device__ __forceinline__ double wide_ldf(const double *p) {
  double v;
  asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// L2 prefetch of a contiguous range, widened to 16-byte granules (the runner's arrays sit in 256-byte aligned slots)
__device__ __forceinline__ void wide_prefetch(const void *p, size_t bytes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~uintptr_t(15);
  const uintptr_t e = (reinterpret_cast<uintptr_t>(p) + bytes + 15) & ~uintptr_t(15);
  if (e > a) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(e - a)) : "memory");
}

// lanes 0..9 of a warp each prefetch one of the streams that a tile reads after its volume products
template <typename T>
__device__ __forceinline__ void wide_prefetch_late(const RhsArgs<T> &A, const Tile &tl, int np, int lane) {
  const size_t nn = (size_t)tl.nelem * np * sizeof(T);
  if (lane < 9) wide_prefetch(A.geo[lane] + tl.node_base, nn);
  else if (lane == 9 && A.resu) wide_prefetch(A.resu + tl.node_base, nn);
}

// lanes 0..5: the streams that a tile reads first
template <typename T>
__device__ __forceinline__ void wide_prefetch_early(const RhsArgs<T> &A, const Tile &tl, int np, int nf, int lane) {
  const size_t fn = (size_t)tl.nelem * nf;
  if (lane < 4) wide_prefetch(A.face[lane] + tl.face_base, fn * sizeof(T));
  else if (lane == 4) wide_prefetch(A.u_in + tl.node_base, (size_t)tl.nelem * np * sizeof(T));
  else if (lane == 5) wide_prefetch(A.gmap + tl.face_base, fn * sizeof(int32_t));
}

// Dr, Ds, Dt times the tile's elements for one m-tile: A fragments (3 per k-step) from ap, DEPTH - 1 k-steps ahead
template <typename C, int NT>
__device__ __forceinline__ void wide_volume(const double *ap, const double *su, int ar, int ac, int conservative,
                                            double (&c)[3][NT][2]) {
  constexpr int KT = C::KT, SU = C::SU, DEPTH = C::DEPTH;
  double f[DEPTH][3];
#pragma unroll
  for (int d = 0; d < DEPTH - 1; ++d)
#pragma unroll
    for (int m = 0; m < 3; ++m) f[d][m] = wide_ldf(ap + d * 96 + m * 32);
#pragma unroll 1
  for (int k0 = 0; k0 < KT; k0 += DEPTH) {
#pragma unroll
    for (int d = 0; d < DEPTH; ++d) {
      const int kk = k0 + d, kn = min(kk + DEPTH - 1, KT - 1);
#pragma unroll
      for (int m = 0; m < 3; ++m) f[(d + DEPTH - 1) % DEPTH][m] = wide_ldf(ap + kn * 96 + m * 32);
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        double bv = su[(8 * n + ar) * SU + 4 * kk + ac];
        if (conservative) bv = 0.5 * bv * bv;
#pragma unroll
        for (int m = 0; m < 3; ++m) wide_dmma(c[m][n][0], c[m][n][1], f[d][m], bv);
      }
    }
  }
}

template <int N, int NT, typename T>
__global__ void __launch_bounds__(WideCfg<N, NT>::THREADS, WideCfg<N, NT>::MINB)
    rhs_stage_wide_kernel(const RhsArgs<T> A, int rhs_only) {
  using C = WideCfg<N, NT>;
  constexpr int NP = C::NP, NF = C::NF, MT = C::MT, KT = C::KT, KL = C::KL, SU = C::SU, SF = C::SF, TE = C::TE;
  constexpr int THREADS = C::THREADS, W = C::WARPS, DEPTH = C::DEPTH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double *su = reinterpret_cast<double *>(smem_raw);  // [TE][SU] state
  double *sv = su + TE * SU;                          // [TE][SU] volume terms
  double *sf = sv + TE * SU;                          // [TE][SF] neighbour traces, then face terms
  int *sfm = reinterpret_cast<int *>(sf + TE * SF);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ar = lane >> 2, ac = lane & 3;
  for (int i = tid; i < NF; i += THREADS) sfm[i] = A.fmask[i];
  pdl_wait();
  if (warp == 0) wide_prefetch_early(A, A.tiles[blockIdx.x], NP, NF, lane);
  const T a = A.a, b = A.b, dt = A.dt;
  __syncthreads();
  for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
    const Tile tl = A.tiles[t];
    const int ne = tl.nelem, nn = ne * NP, nfc = ne * NF;
    if (tid == 0 && t + (int)gridDim.x >= A.ntiles) pdl_trigger();
    // state, and neighbour traces of this thread's face points (index batch, then gather batch)
    constexpr int CH = 4;
    for (int x0 = tid; x0 < nn; x0 += CH * THREADS) {
      T v[CH];
#pragma unroll
      for (int j = 0; j < CH; ++j) v[j] = x0 + j * THREADS < nn ? A.u_in[tl.node_base + x0 + j * THREADS] : T(0);
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int x = x0 + j * THREADS, e = x / NP;
        if (x < nn) su[e * SU + x - e * NP] = v[j];
      }
    }
    __syncthreads();
    for (int x0 = tid; x0 < nfc; x0 += CH * THREADS) {
      int32_t src[CH];
      T up[CH], fc[CH][4];
#pragma unroll
      for (int j = 0; j < CH; ++j) src[j] = x0 + j * THREADS < nfc ? __ldcs(A.gmap + tl.face_base + x0 + j * THREADS) : 0;
#pragma unroll
      for (int j = 0; j < CH; ++j)
#pragma unroll
        for (int m = 0; m < 4; ++m)
          fc[j][m] = x0 + j * THREADS < nfc ? __ldcs(A.face[m] + tl.face_base + x0 + j * THREADS) : T(0);
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const bool ok = src[j] >= 0 && (int64_t)src[j] < A.n_u_values;
        up[j] = ok ? A.u_in[src[j]] : T(0);
      }
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int x = x0 + j * THREADS;
        if (x < nfc) {
          const int e = x / NF, q = x - e * NF;
          const T uM = (T)su[e * SU + sfm[q]];
          T uP = up[j];
          if (!(src[j] >= 0 && (int64_t)src[j] < A.n_u_values)) {  // rejected index: report it, use the interior trace
            atomicExch(A.status, kStatusBadGather);
            uP = uM;
          }
          const T nsum = fc[j][0] + fc[j][1] + fc[j][2];
          const T fM = T(0.5) * uM * uM * nsum, fP = T(0.5) * uP * uP * nsum;
          const T an = fabs(nsum);
          const T lam = fmax(fabs(uM) * an, fabs(uP) * an);
          sf[e * SF + q] = fc[j][3] * (fM - (T(0.5) * (fM + fP) + T(0.5) * lam * (uM - uP)));
        }
      }
    }
    if (warp == 0) wide_prefetch_late(A, tl, NP, lane);
#pragma unroll 1
    for (int mt = warp; mt < MT; mt += W) {
      const double *ap = A.D64 + (size_t)mt * KT * 96 + lane;
      double c[3][NT][2];
#pragma unroll
      for (int m = 0; m < 3; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) c[m][n][0] = c[m][n][1] = 0.0;
      wide_volume<C, NT>(ap, su, ar, ac, A.conservative, c);
      const int row = 8 * mt + ar;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        T g[2][9];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 8 * n + 2 * ac + h;
#pragma unroll
          for (int m = 0; m < 9; ++m)
            g[h][m] = (row < NP && e < ne) ? __ldcs(A.geo[m] + tl.node_base + e * NP + row) : 0.0;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 8 * n + 2 * ac + h;
          const T ur = (T)c[0][n][h], us = (T)c[1][n][h], ut = (T)c[2][n][h];
          const T ux = g[h][0] * ur + g[h][3] * us + g[h][6] * ut;
          const T uy = g[h][1] * ur + g[h][4] * us + g[h][7] * ut;
          const T uz = g[h][2] * ur + g[h][5] * us + g[h][8] * ut;
          if (row < NP && e < ne) sv[e * SU + row] = A.conservative ? -(ux + uy + uz) : -(T)su[e * SU + row] * (ux + uy + uz);
        }
      }
    }
    __syncthreads();  // face terms complete
    if (warp == W - 1 && t + (int)gridDim.x < A.ntiles) wide_prefetch_early(A, A.tiles[t + gridDim.x], NP, NF, lane);
    // LIFT times the face terms, then the update; each lane reads back the volume terms it wrote
#pragma unroll 1
    for (int mt = warp; mt < MT; mt += W) {
      const double *ap = A.L64 + (size_t)mt * KL * 32 + lane;
      const int row = 8 * mt + ar;
      double c[NT][2];
      T rs[NT][2];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 8 * n + 2 * ac + h;
          c[n][h] = 0.0;
          rs[n][h] = (!rhs_only && row < NP && e < ne) ? __ldcs(A.resu + tl.node_base + e * NP + row) : T(0);
        }
      double f[4];
#pragma unroll
      for (int d = 0; d < 3; ++d) f[d] = wide_ldf(ap + d * 32);
#pragma unroll 1
      for (int k0 = 0; k0 < KL; k0 += 4) {
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          const int kk = k0 + d;
          f[(d + 3) % 4] = wide_ldf(ap + min(kk + 3, KL - 1) * 32);
#pragma unroll
          for (int n = 0; n < NT; ++n) wide_dmma(c[n][0], c[n][1], f[d], sf[(8 * n + ar) * SF + 4 * kk + ac]);
        }
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 8 * n + 2 * ac + h;
          if (row < NP && e < ne) {
            const int64_t gi = tl.node_base + e * NP + row;
            const T rhs = (T)sv[e * SU + row] + (T)c[n][h];
            if (rhs_only) {
              __stcs(A.rhs_out + gi, rhs);
            } else {
              const T res = a * rs[n][h] + dt * rhs;
              __stcs(A.resu + gi, res);
              __stcs(A.u_out + gi, (T)su[e * SU + row] + b * res);
            }
          }
        }
    }
    __syncthreads();  // the tile's buffers are free
  }
}

// Volume derivative (mode 0) and the reference's volume-only right-hand side (mode 1): the same products, results
// stored from the epilogue.
template <int N, int NT, typename T>
__global__ void __launch_bounds__(WideCfg<N, NT>::THREADS, WideCfg<N, NT>::MINB) diff_wide_kernel(const DiffArgs<T> A) {
  using C = WideCfg<N, NT>;
  constexpr int NP = C::NP, MT = C::MT, KT = C::KT, SU = C::SU, TE = C::TE, THREADS = C::THREADS, W = C::WARPS;
  __shared__ double su[TE * SU];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ar = lane >> 2, ac = lane & 3;
  pdl_wait();
  for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
    const Tile tl = A.tiles[t];
    const int ne = tl.nelem, nn = ne * NP;
    if (tid == 0 && t + (int)gridDim.x >= A.ntiles) pdl_trigger();
    constexpr int CH = 4;
    for (int x0 = tid; x0 < nn; x0 += CH * THREADS) {
      T v[CH];
#pragma unroll
      for (int j = 0; j < CH; ++j) v[j] = x0 + j * THREADS < nn ? __ldcs(A.u + tl.node_base + x0 + j * THREADS) : T(0);
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        const int x = x0 + j * THREADS, e = x / NP;
        if (x < nn) su[e * SU + x - e * NP] = v[j];
      }
    }
    if (warp == 0 && lane < 9) wide_prefetch(A.geo[lane] + tl.node_base, (size_t)nn * sizeof(T));
    __syncthreads();
#pragma unroll 1
    for (int mt = warp; mt < MT; mt += W) {
      double c[3][NT][2] = {};
      wide_volume<C, NT>(A.D64 + (size_t)mt * KT * 96 + lane, su, ar, ac, 0, c);
      const int row = 8 * mt + ar;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        T g[2][9];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 8 * n + 2 * ac + h;
#pragma unroll
          for (int m = 0; m < 9; ++m)
            g[h][m] = (row < NP && e < ne) ? __ldcs(A.geo[m] + tl.node_base + e * NP + row) : T(0);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = 8 * n + 2 * ac + h;
          if (row < NP && e < ne) {
            const int64_t gi = tl.node_base + e * NP + row;
            const T ur = (T)c[0][n][h], us = (T)c[1][n][h], ut = (T)c[2][n][h];
            const T ux = g[h][0] * ur + g[h][3] * us + g[h][6] * ut;
            const T uy = g[h][1] * ur + g[h][4] * us + g[h][7] * ut;
            const T uz = g[h][2] * ur + g[h][5] * us + g[h][8] * ut;
            if (A.mode == 0) {
              __stcs(A.out[0] + gi, ux);
              __stcs(A.out[1] + gi, uy);
              __stcs(A.out[2] + gi, uz);
            } else {
              A.out[0][gi] = -(T)su[e * SU + row] * (ux + uy + uz);  // not streamed: an update reads it next
            }
          }
        }
      }
    }
    __syncthreads();  // the tile's buffer is free
  }
}

template <int N, int NT, typename T>
void wide_diff_n(const DiffArgs<T> &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  using C = WideCfg<N, NT>;
  auto k = diff_wide_kernel<N, NT, T>;
  const int per = resident_ctas(k, C::THREADS, 0, info);
  const int grid = std::min(A.ntiles, per * num_sms);
  if (info) *info = {grid, C::THREADS, 0, per};
  if (grid > 0) launch_pdl(k, grid, C::THREADS, 0, st, A);
}

template <int N, int NT, typename T>
void wide_launch_n(const RhsArgs<T> &A, int rhs_only, int num_sms, cudaStream_t st, LaunchInfo *info) {
  using C = WideCfg<N, NT>;
  auto k = rhs_stage_wide_kernel<N, NT, T>;
  const int per = resident_ctas(k, C::THREADS, C::SMEM, info);
  const int grid = std::min(A.ntiles, per * num_sms);
  if (info) *info = {grid, C::THREADS, (int)C::SMEM, per};
  if (grid > 0) launch_pdl(k, grid, C::THREADS, C::SMEM, st, A, rhs_only);
}

}  // namespace

bool wide_supported(int N) { return N == 6 || N == 7; }

// Tiles of 16 elements reuse a matrix fragment twice; below two such tiles per SM, tiles of 8 keep more SMs busy.
int wide_tile_elems(int64_t nelems, int num_sms) {
  return (nelems + 15) / 16 >= 2 * (int64_t)num_sms ? 16 : 8;
}

std::vector<double> wide_pack(const std::vector<double> &mats, int nmats, int rows, int cols) {
  const int mt = (rows + 7) / 8, kt = cols / 4;
  std::vector<double> out((size_t)mt * kt * nmats * 32, 0.0);
  for (int t = 0; t < mt; ++t)
    for (int k = 0; k < kt; ++k)
      for (int m = 0; m < nmats; ++m)
        for (int l = 0; l < 32; ++l) {
          const int i = 8 * t + (l >> 2), j = 4 * k + (l & 3);
          if (i < rows) out[(((size_t)t * kt + k) * nmats + m) * 32 + l] = mats[((size_t)m * rows + i) * cols + j];
        }
  return out;
}

template <typename T>
void launch_rhs_wide(int N, int tile_elems, const RhsArgs<T> &A, int rhs_only, int num_sms, cudaStream_t st,
                     LaunchInfo *info) {
  const int nt = tile_elems / 8;
  if (N == 6 && nt == 2) wide_launch_n<6, 2, T>(A, rhs_only, num_sms, st, info);
  else if (N == 6 && nt == 1) wide_launch_n<6, 1, T>(A, rhs_only, num_sms, st, info);
  else if (N == 7 && nt == 2) wide_launch_n<7, 2, T>(A, rhs_only, num_sms, st, info);
  else if (N == 7 && nt == 1) wide_launch_n<7, 1, T>(A, rhs_only, num_sms, st, info);
  else throw Error(DGK_ERR_UNSUPPORTED, "wide FP64 stage: orders 6 and 7, tiles of 8 or 16 elements");
}

template <typename T>
void launch_diff_wide(int N, int tile_elems, const DiffArgs<T> &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  const int nt = tile_elems / 8;
  if (N == 6 && nt == 2) wide_diff_n<6, 2, T>(A, num_sms, st, info);
  else if (N == 6 && nt == 1) wide_diff_n<6, 1, T>(A, num_sms, st, info);
  else if (N == 7 && nt == 2) wide_diff_n<7, 2, T>(A, num_sms, st, info);
  else if (N == 7 && nt == 1) wide_diff_n<7, 1, T>(A, num_sms, st, info);
  else throw Error(DGK_ERR_UNSUPPORTED, "wide derivative: orders 6 and 7, tiles of 8 or 16 elements");
}

template void launch_diff_wide<double>(int, int, const DiffArgs<double> &, int, cudaStream_t, LaunchInfo *);
template void launch_diff_wide<float>(int, int, const DiffArgs<float> &, int, cudaStream_t, LaunchInfo *);
template void launch_rhs_wide<double>(int, int, const RhsArgs<double> &, int, int, cudaStream_t, LaunchInfo *);
template void launch_rhs_wide<float>(int, int, const RhsArgs<float> &, int, int, cudaStream_t, LaunchInfo *);

}  // namespace dgk
