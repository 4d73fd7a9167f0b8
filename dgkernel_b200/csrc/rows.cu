// Mixed-precision stage with a matrix row per thread: order 1, and orders 2..4 while a problem is small (operator
// "rhsStageMixed"; the arithmetic is mixed.cu's, bit for bit: compensated pair state, products on the field minus its
// linear vertex interpolant, flux and residual in FP32, update in FP64).
//
// mixed.cu gives each lane an element, which amortises the work around the products but leaves a small problem as a
// few long serial chains: 12 us for any order-3 problem of up to 10,000 elements.  Here a thread owns one output row:
// its rows of Dr, Ds, Dt and LIFT stay in registers for the whole persistent kernel (100 values at order 3), and the
// element vectors are read from shared memory as 16-byte broadcasts, four columns of three matrices (six paired FMAs)
// per load.  Thread (e, i) also owns node i of element e and the face points i, i + Np, ...: consecutive threads are
// consecutive values in memory, so state, residual, gather map and results move as coalesced loads and stores with no
// staging.  Everything a tile reads is loaded into registers a tile ahead (the neighbour traces, whose indices are
// loaded two tiles ahead, straight from L2), and the shared-memory buffers alternate, so a tile has two barriers: the
// tile's state is stored; its operands (field minus linear part, face terms) are.  Bound by its instruction count (about
// 330 per node at order 3 against mixed.cu's 150) once every SM is busy.  The lines of rows_faster follow from stages in
// a captured graph, us, mixed.cu / here:
//   elements    order 1       order 2        order 3      order 4
//        384    3.8 / 1.9     6.2 / 2.7      9.5 / 3.3   18.9 / 6.0
//       6000    5.4 / 2.3     8.1 / 3.9     11.9 / 6.8   21.7 / 10.7
//      16464    6.0 / 2.9     8.7 / 6.2     12.1 / 10.5  22.3 / 20.6
//      20250                  8.9 / 6.6     12.8 / 11.5  25.2 / 24.2
//      24576                  9.6 / 7.0     14.2 / 13.6  27.1 / 28.3
//      29478    7.2 / 2.9     9.9 / 8.1     14.4 / 15.4  27.6 / 33.3
//      48000    8.7 / 4.2    11.9 / 10.7
//      82944                 16.2 / 15.8
//      93750                 17.2 / 17.7
//     131712   15.4 / 8.0    22.0 / 24.1    39.1 / 58.0  87.0 / 127.6
//     384000   37.7 / 19.5   52.5 / 68.8
//     663552   62.7 / 32.1   87.6 / 119.6
#include <algorithm>
#include <cstdint>

#include "dg_kernels.cuh"
#include "launch.cuh"

namespace dgk {

namespace {

template <int N>
struct RowCfg {
  using O = Order<N>;
  static constexpr int NP = O::NP, NFP = O::NFP, NF = O::NF;
  static constexpr int NPJ = (NP + 3) & ~3;  // columns padded to whole float4 groups
  static constexpr int EP = N == 1 ? 32 : N == 2 ? 16 : N == 3 ? 6 : 7;  // elements side by side (whole warps nearly)
  static constexpr int G = 2, TE = EP * G;                  // element groups, elements per tile
  static constexpr int THREADS = (EP * NP + 31) / 32 * 32;
  static constexpr int NJ = (NF + NP - 1) / NP;             // face points per thread and element
  static constexpr int NG = (TE * kMixedGeoWords + THREADS - 1) / THREADS;
  static constexpr int MINB = N == 1 ? 4 : N == 4 ? 1 : 3;  // by registers: 128, 128, 168, 255 a thread
  static_assert(NF % 4 == 0, "face terms are read as float4");
};

template <int N>
struct RowSmem {
  using C = RowCfg<N>;
  float dw[2][C::TE * C::NPJ];           // field minus its linear part
  float fl[2][C::TE * C::NF];            // face terms
  float geo[2][C::TE * kMixedGeoWords];  // compact geometry; the pad word takes the linear part's derivative
  double u[2][C::TE * C::NP];
  float hi[2][C::TE * C::NP];
};

// The field whose derivative is taken: u or u^2/2, rounded by itself (a product that the compiler may merge with the
// subtraction after it would leave mixed.cu's bits, whose form is chosen at run time).
template <bool CONS>
__device__ __forceinline__ double row_w(double u) {
  return CONS ? __dmul_rn(0.5 * u, u) : u;
}

template <int N, bool CONS>
__global__ void __launch_bounds__(RowCfg<N>::THREADS, RowCfg<N>::MINB) rhs_stage_rows_kernel(const MixedArgs A) {
  using C = RowCfg<N>;
  constexpr int NP = C::NP, NFP = C::NFP, NF = C::NF, NPJ = C::NPJ, EP = C::EP, G = C::G, TE = C::TE, NJ = C::NJ;
  constexpr int THREADS = C::THREADS, NG = C::NG;
  __shared__ __align__(16) RowSmem<N> m;
  const int tid = threadIdx.x, step = gridDim.x, ntiles = A.ntiles;
  const bool lives = tid < EP * NP;  // the last warp's spare lanes mirror element 0's first row and store nothing
  const int ep = lives ? tid / NP : 0, i = lives ? tid - ep * NP : 0;
  for (int x = tid; x < 2 * TE * NPJ; x += THREADS) (&m.dw[0][0])[x] = 0.f;  // padded columns stay zero
  const int vA = A.vtx[0], vB = A.vtx[1], vC = A.vtx[2], vD = A.vtx[3];
  const double b1 = A.bary[3 * i], b2 = A.bary[3 * i + 1], b3 = A.bary[3 * i + 2];
  int fm[NJ], fg[NJ];  // this thread's face points: interior node, geometry word of the face
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    const int q = min(i + NP * j, NF - 1);
    fm[j] = A.fmask[q];
    fg[j] = 3 + q / NFP;
  }
  float2 D[3][NPJ / 2], L[NF / 2];
#pragma unroll
  for (int j = 0; j < NPJ / 2; ++j)
#pragma unroll
    for (int d = 0; d < 3; ++d) D[d][j] = *reinterpret_cast<const float2 *>(A.Dm + i * 3 * NPJ + j * 6 + d * 2);
#pragma unroll
  for (int j = 0; j < NF / 2; ++j) L[j] = *reinterpret_cast<const float2 *>(A.lift + i * NF + 2 * j);
  const float a = A.a, dt = A.dt;
  const double b = A.b;
  const uint32_t nvalues = (uint32_t)A.n_u_values;

  // next tile's state, residual, geometry and neighbour traces; gather indices of the tile after it
  float nh[G], nl[G], nr[G], ng[NG], up[G][NJ];
  int32_t idx[G][NJ];
  uint32_t bad = 0;  // points whose index is out of range (the interior trace stands)
  const int po = ep * NF + i, no = ep * NP + i;  // first face point and node of this thread within a tile
  auto load_idx = [&](const MTile &tl) {
    const int32_t *gm = A.gmap + tl.face_base + po;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const bool in = g * EP + ep < tl.nelem;
#pragma unroll
      for (int j = 0; j < NJ; ++j) idx[g][j] = (in && i + NP * j < NF) ? __ldcs(gm + g * EP * NF + NP * j) : 0;
    }
  };
  auto load_tile = [&](const MTile &tl) {
    bad = 0;
    const float *hp = A.uhi_in + tl.node_base + no, *lp = A.ulo_in + tl.node_base + no, *rp = A.resu + tl.node_base + no;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const bool in = g * EP + ep < tl.nelem;  // (a spare lane mirrors a thread that lives)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const bool ok = (uint32_t)idx[g][j] < nvalues;
        if (!ok) bad |= 1u << (g * NJ + j);
        up[g][j] = ok ? __ldcg(A.uhi_in + (uint32_t)idx[g][j]) : 0.f;
      }
      nh[g] = in ? __ldcg(hp + g * EP * NP) : 0.f;
      nl[g] = in ? __ldcs(lp + g * EP * NP) : 0.f;
      nr[g] = in ? __ldcs(rp + g * EP * NP) : 0.f;
    }
    const float *gp = A.geo + tl.elem_slot * kMixedGeoWords + tid;
#pragma unroll
    for (int j = 0; j < NG; ++j)
      ng[j] = tid + j * THREADS < tl.nelem * kMixedGeoWords ? __ldcs(gp + j * THREADS) : 0.f;
    if (bad) atomicExch(A.status, kStatusBadGather);
  };
  MTile t0 = A.tiles[blockIdx.x], t1{}, t2{};
  pdl_wait();
  load_idx(t0);
  load_tile(t0);
  if (blockIdx.x + step < ntiles) {
    t1 = A.tiles[blockIdx.x + step];
    load_idx(t1);
  }
  if (blockIdx.x + 2 * step < ntiles) t2 = A.tiles[blockIdx.x + 2 * step];
  __syncthreads();
  int p = 0;
  for (int t = blockIdx.x; t < ntiles; t += step, p ^= 1) {
    const int ne = t0.nelem;
    if (tid == 0 && t + step >= ntiles) pdl_trigger();
    // (1) the tile's state and geometry into shared memory
    double u[G];
    float h[G], r[G], uP[G][NJ];
    const uint32_t rejected = bad;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      h[g] = nh[g];
      r[g] = nr[g];
      u[g] = (double)nh[g] + (double)nl[g];
#pragma unroll
      for (int j = 0; j < NJ; ++j) uP[g][j] = up[g][j];
      if (lives) {
        m.u[p][g * EP * NP + no] = u[g];
        m.hi[p][g * EP * NP + no] = h[g];
      }
    }
#pragma unroll
    for (int j = 0; j < NG; ++j)
      if (tid + j * THREADS < TE * kMixedGeoWords) m.geo[p][tid + j * THREADS] = ng[j];
    __syncthreads();
    // loads of the next tile, and of the gather indices and descriptor after it, in flight from here on
    MTile t3{};
    if (t + step < ntiles) load_tile(t1);
    if (t + 2 * step < ntiles) load_idx(t2);
    if (t + 3 * step < ntiles) t3 = A.tiles[t + 3 * step];
    // (2) operands: field minus its linear interpolant through the vertex nodes (FP64), and the Lax-Friedrichs
    // surface term times Fscale: 1/2 (uM-uP) (1/2 (uM+uP) g - max(|uM|,|uP|) |g|)
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int e = g * EP + ep;
      const double *ue = m.u[p] + e * NP;
      const float *ge = m.geo[p] + e * kMixedGeoWords, *he = m.hi[p] + e * NP;
      const double uA = ue[vA], uB = ue[vB], uC = ue[vC], uD = ue[vD];
      const double wA = row_w<CONS>(uA), w = row_w<CONS>(u[g]);
      const double dB = row_w<CONS>(uB) - wA, dC = row_w<CONS>(uC) - wA, dD = row_w<CONS>(uD) - wA;
      if (lives) m.dw[p][e * NPJ + i] = (float)((w - wA) - (b1 * dB + b2 * dC + b3 * dD));
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const float gq = ge[fg[j]], uM = he[fm[j]];
        const float v = ((rejected >> (g * NJ + j)) & 1u) ? uM : uP[g][j];
        const float d = uM - v;
        const float fl = 0.5f * d * (0.5f * (uM + v) * gq - fmaxf(fabsf(uM), fabsf(v)) * fabsf(gq));
        if (lives && i + NP * j < NF) m.fl[p][g * EP * NF + po + NP * j] = fl;
      }
    }
    if (tid < TE) {
      // derivative of the linear part along (1,1,1), one thread per element: d/dr = (wB-wA)/2 and likewise for s, t
      const double *ue = m.u[p] + tid * NP;
      float *ge = m.geo[p] + tid * kMixedGeoWords;
      const double wA = row_w<CONS>(ue[vA]);
      const double dB = row_w<CONS>(ue[vB]) - wA, dC = row_w<CONS>(ue[vC]) - wA, dD = row_w<CONS>(ue[vD]) - wA;
      ge[7] = (float)(0.5 * ((double)ge[0] * dB + (double)ge[1] * dC + (double)ge[2] * dD));
    }
    __syncthreads();
    // (3) products of this thread's row with each of its elements, stage update
    float *hp = A.uhi_out + t0.node_base + no, *lp = A.ulo_out + t0.node_base + no, *rp = A.resu + t0.node_base + no;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int e = g * EP + ep;
      const float4 *x4 = reinterpret_cast<const float4 *>(m.dw[p] + e * NPJ);
      float2 ar = make_float2(0.f, 0.f), as = ar, at = ar, br = ar, bs = ar, bt = ar;
#pragma unroll
      for (int k = 0; k < NPJ / 4; ++k) {
        const float4 x = x4[k];
        const float2 xa = make_float2(x.x, x.y), xb = make_float2(x.z, x.w);
        ar = __ffma2_rn(D[0][2 * k], xa, ar);
        as = __ffma2_rn(D[1][2 * k], xa, as);
        at = __ffma2_rn(D[2][2 * k], xa, at);
        br = __ffma2_rn(D[0][2 * k + 1], xb, br);
        bs = __ffma2_rn(D[1][2 * k + 1], xb, bs);
        bt = __ffma2_rn(D[2][2 * k + 1], xb, bt);
      }
      const float ur = (ar.x + ar.y) + (br.x + br.y);
      const float us = (as.x + as.y) + (bs.x + bs.y);
      const float ut = (at.x + at.y) + (bt.x + bt.y);
      const float4 ga = *reinterpret_cast<const float4 *>(m.geo[p] + e * kMixedGeoWords);
      const float L0 = m.geo[p][e * kMixedGeoWords + 7];
      const float dd = fmaf(ga.x, ur, fmaf(ga.y, us, fmaf(ga.z, ut, L0)));
      const float vol = CONS ? -dd : -h[g] * dd;
      const float4 *f4 = reinterpret_cast<const float4 *>(m.fl[p] + e * NF);
      float2 l0 = make_float2(0.f, 0.f), l1 = l0, l2 = l0, l3 = l0;
#pragma unroll
      for (int k = 0; k < NF / 4; ++k) {
        const float4 x = f4[k];
        if (k & 1) {
          l2 = __ffma2_rn(L[2 * k], make_float2(x.x, x.y), l2);
          l3 = __ffma2_rn(L[2 * k + 1], make_float2(x.z, x.w), l3);
        } else {
          l0 = __ffma2_rn(L[2 * k], make_float2(x.x, x.y), l0);
          l1 = __ffma2_rn(L[2 * k + 1], make_float2(x.z, x.w), l1);
        }
      }
      const float lift = ((l0.x + l0.y) + (l1.x + l1.y)) + ((l2.x + l2.y) + (l3.x + l3.y));
      const float rn = fmaf(dt, lift, fmaf(a, r[g], dt * vol));
      const double un = u[g] + b * (double)rn;
      const float hn = __double2float_rn(un);
      if (lives && e < ne) {
        hp[g * EP * NP] = hn;
        __stcs(lp + g * EP * NP, __double2float_rn(un - (double)hn));
        __stcs(rp + g * EP * NP, rn);
      }
    }
    t0 = t1;
    t1 = t2;
    t2 = t3;
  }
}

template <int N, bool CONS>
void rows_launch_n(const MixedArgs &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  using C = RowCfg<N>;
  const int per = resident_ctas(rhs_stage_rows_kernel<N, CONS>, C::THREADS, 0, info);
  const int grid = std::min(A.ntiles, per * num_sms);
  if (info) *info = {grid, C::THREADS, (int)sizeof(RowSmem<N>), per};
  if (grid > 0) launch_pdl(rhs_stage_rows_kernel<N, CONS>, grid, C::THREADS, 0, st, A);
}

template <int N>
void rows_launch(const MixedArgs &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  if (A.conservative)
    rows_launch_n<N, true>(A, num_sms, st, info);
  else
    rows_launch_n<N, false>(A, num_sms, st, info);
}

}  // namespace

int rows_tile_elems(int N) {
  switch (N) {
    case 1: return RowCfg<1>::TE;
    case 2: return RowCfg<2>::TE;
    case 3: return RowCfg<3>::TE;
    case 4: return RowCfg<4>::TE;
    default: return 0;
  }
}

// Elements per SM up to which this form is taken (148 SMs; the table above): order 1 always, orders 2 and 3 up to their
// crossings, order 4 somewhat below it.
bool rows_faster(int N, int64_t nelems, int num_sms) {
  switch (N) {
    case 1: return true;
    case 2: return nelems <= 590 * (int64_t)num_sms;
    case 3: return nelems <= 175 * (int64_t)num_sms;
    case 4: return nelems <= 110 * (int64_t)num_sms;
    default: return false;
  }
}

void launch_rhs_rows(int N, const MixedArgs &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  switch (N) {
    case 1: rows_launch<1>(A, num_sms, st, info); break;
    case 2: rows_launch<2>(A, num_sms, st, info); break;
    case 3: rows_launch<3>(A, num_sms, st, info); break;
    case 4: rows_launch<4>(A, num_sms, st, info); break;
    default: throw Error(DGK_ERR_UNSUPPORTED, "row form of the mixed stage: orders 1..4");
  }
}

}  // namespace dgk
