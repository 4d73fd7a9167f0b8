// Learned-sensor artificial viscosity on the mixed-precision stage: the shock sensor over every element, then
// the BR1 viscous term only where it is not zero.
//
// Per stage, before the tensor-core mixed stage (tcm.cu), which adds the result to its right-hand side:
//   ls_sensor   every element: modal coefficients uhat = Vinv u (FP64, on the FP64 tensor path), the
//               Persson-Peraire activation from log10(E_top / E), the 35 -> 32 -> 32 -> 1 network (tanh, tanh,
//               sigmoid; FP16 weights, FP32 sums; its hidden layers as FP16 tensor products with two-part
//               inputs) on uhat / |uhat| with the PP fallback inside (lo, hi) and, in mode 3, outputs <= lo read
//               as a smooth element; eps_e = eps0 sigma_e h_e / N; elements with eps_e > 0 form the active list.
//               The pass marks the active elements and their face neighbours, and ls_compact lists them (touched).
//   ls_grad     active elements: q_d = D_d u + LIFT (Fscale n_d (uP - uM) / 2) (FP64 tensor path), stored as
//               eps_e q_d.
//   ls_div      touched elements: sum_d d/dx_d (eps_e q_d) + LIFT (Fscale / 2 sum_d n_d (epsP qP_d - epsM qM_d)),
//               the viscous right-hand side, with eps q = 0 on elements that are not active; on straight-sided
//               elements the derivative is sum_k D_k (sum_d (d xi_k / d x_d) eps q_d) (FP64 tensor path).
// This is the BR1 viscosity of the plain viscosity stage (av.cu) restricted to where it is not zero: an element
// whose own and neighbours' eps vanish gets no viscous term there either.  The sparse passes walk device-side
// counts with persistent grids, so a stage needs no host synchronisation.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>

#include "dg_kernels.cuh"
#include "launch.cuh"

namespace dgk {

namespace {

constexpr int kLsHid = 32;
constexpr int kLsWarps = 8;  // sensor pass: warps per block, 8 elements each at a time

__device__ __forceinline__ double ls_pp_sigma(double S, double s0, double kappa) {
  if (!(S >= s0 - kappa)) return 0.0;
  if (S > s0 + kappa) return 1.0;
  return 0.5 * (1.0 + sin(3.141592653589793 * (S - s0) / (2.0 * kappa)));
}

// partition of an element slot (slot_prefix ascending)
__device__ __forceinline__ int part_of_slot(const LsArgs &A, int64_t slot) {
  int p = 0;
  while (p + 1 < A.npart && A.slot_prefix[p + 1] <= slot) ++p;
  return p;
}

// element slot and local node of a state value index; -1 when it lies in no partition
__device__ __forceinline__ int64_t slot_of_value(const LsArgs &A, int64_t g, int np, int *node) {
  for (int p = 0; p < A.npart; ++p) {
    const int64_t rel = g - A.uoff[p];
    if (rel >= 0 && rel < A.kpart[p] * np) {
      const int64_t le = rel / np;
      *node = (int)(rel - le * np);
      return A.slot_prefix[p] + le;
    }
  }
  *node = 0;
  return -1;
}

// The network's inputs as FP16 pairs: x 2^15 = hi + lo 2^-11, both rounded to nearest (|x| <= 1: a unit-norm feature or a
// tanh).  The largest error is 1.2e-7 of x down to x = 2e-9, what a pair of TF32 parts has, and 4.4e-16 below, where the
// state's pair and the modal transform carry x no further: the scales keep both parts out of FP16's subnormals, which is
// why the low products have sums of their own (both parts at 2^10: 2.9e-6 of x at 1e-5 and 2.9e-3 at 1e-8).
constexpr float kLsScale = 32768.f, kLsLow = 2048.f;
__device__ __forceinline__ void ls_put(__half *row, int lo_off, float x) {
  const float v = x * kLsScale;
  const __half h = __float2half_rn(v);
  row[0] = h;
  row[lo_off] = __float2half_rn((v - __half2float(h)) * kLsLow);
}

// one m16n8k16 product accumulated into d
__device__ __forceinline__ void ls_mma_f16(float (&d)[4], const uint4 &a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ls_dmma(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Sensor pass.  Each warp walks its own groups of 8 elements with no block barrier; the next group's state, first slot
// and h / N are loaded while the current one is computed.  Lane (g = l / 4, c = l mod 4) of the tensor products holds
// output rows g, g + 8, ... of elements 2c and 2c + 1, so the energies are summed and the features formed straight from
// the accumulators, and every lane ends with one element: 2c + (g mod 2).  Shared memory is what bounds the pass (its
// pipe was 85 % busy with the matrix and the weights read entry by entry and rows at conflicting strides), so Vinv and
// the weights lie there in fragment order (one 8-byte load per lane and fragment) and the rows at strides that spread
// the 8 rows of a fragment over the banks.  The logarithm and the sine of the ramp run only where the energy ratio can
// reach it.  Order 4, 32^3 x 6: 75 us with entry-by-entry reads, 61 so, 57 with the network on FP16 pairs (half the
// products of TF32 ones at the same 22 bits an input, and the weights need no conversion).
template <int N>
struct LsSensorSmem {
  static constexpr int NP = Order<N>::NP, MT = (NP + 7) / 8, KT = (NP + 3) / 4, K1 = (NP + 15) / 16, K2 = kLsHid / 16;
  static constexpr int SU = frag_stride(NP);           // nodal values of an element
  static constexpr int SX = 8 * K1 + 4;  // words of a feature row: two FP16 each, 4 mod 8 (conflict-free)
  static constexpr int SH = 8 * K2 + 4;                // words of a row of hidden units
  double vinv[MT * KT * 32];                           // [m-tile][k-step][lane]
  double u[kLsWarps][8 * SU];
  uint4 w[(K1 + K2) * 2 * 32];                         // FP16 weights: [k-step][m-tile][lane], 8 per lane
  uint32_t x[kLsWarps][2][8 * SX], h[kLsWarps][2][8 * SH];  // high and low parts; columns past the inputs stay zero
  float b1[kLsHid], b2[kLsHid], w3[kLsHid], b3;
};

// one hidden layer: o[m-tile] += W x over K k-steps; x points at this lane's word of its element's row, the low
// parts lie `lo` words behind
template <int K>
__device__ __forceinline__ void ls_layer(const uint4 *w, const uint32_t *x, int lo, float (&o)[2][4]) {
  float ol[2][4] = {};  // the low parts' sums, 2^11 times their share
#pragma unroll
  for (int kk = 0; kk < K; ++kk) {
    const uint32_t h0 = x[8 * kk], h1 = x[8 * kk + 4], l0 = x[lo + 8 * kk], l1 = x[lo + 8 * kk + 4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      const uint4 a = w[(kk * 2 + mt) * 32];
      ls_mma_f16(o[mt], a, h0, h1);
      ls_mma_f16(ol[mt], a, l0, l1);
    }
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int f = 0; f < 4; ++f) o[mt][f] = fmaf(ol[mt][f], 1.f / kLsLow, o[mt][f]);
}

template <int N>
__global__ void __launch_bounds__(32 * kLsWarps, 3) ls_sensor_kernel(const LsArgs A) {
  using S = LsSensorSmem<N>;
  constexpr int NP = S::NP, MT = S::MT, KT = S::KT, SU = S::SU, SX = S::SX, SH = S::SH, K1 = S::K1, K2 = S::K2;
  extern __shared__ __align__(16) unsigned char sm[];
  S &m = *reinterpret_cast<S *>(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, c = lane & 3;
  for (int i = tid; i < MT * KT * 32; i += blockDim.x) {
    const int l = i & 31, kk = (i >> 5) % KT, mt = (i >> 5) / KT, r = 8 * mt + (l >> 2), j = 4 * kk + (l & 3);
    m.vinv[i] = (r < NP && j < NP) ? A.Vinv[r * NP + j] : 0.0;
  }
  uint32_t topmask = 0;  // of this lane's rows, those of modes of total degree N
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
    if (8 * mt + g < NP && A.top[8 * mt + g]) topmask |= 1u << mt;
  pdl_wait();
  if (A.mode >= 2) {
    // the network's parameters, rounded to FP16
    const float *W1 = A.mlp, *B1 = W1 + kLsHid * NP, *W2 = B1 + kLsHid, *B2 = W2 + kLsHid * kLsHid, *W3 = B2 + kLsHid;
    auto h16 = [](float v) { return __half2float(__float2half_rn(v)); };
    for (int i = tid; i < (K1 + K2) * 2 * 32; i += blockDim.x) {
      const int l = i & 31, mt = (i >> 5) & 1, kk = i >> 6;
      const bool first = kk < K1;
      const float *W = first ? W1 : W2;
      const int nin = first ? NP : kLsHid, r = 16 * mt + (l >> 2), j = 16 * (first ? kk : kk - K1) + 2 * (l & 3);
      auto pair = [&](int rr, int jj) {
        const __half2 v = __floats2half2_rn(jj < nin ? W[rr * nin + jj] : 0.f, jj + 1 < nin ? W[rr * nin + jj + 1] : 0.f);
        return *reinterpret_cast<const uint32_t *>(&v);
      };
      m.w[i] = make_uint4(pair(r, j), pair(r + 8, j), pair(r, j + 8), pair(r + 8, j + 8));
    }
    for (int i = tid; i < kLsWarps * 2 * 8 * S::SX; i += blockDim.x) (&m.x[0][0][0])[i] = 0;
    if (tid < kLsHid) {
      m.b1[tid] = h16(B1[tid]) * kLsScale;
      m.b2[tid] = h16(B2[tid]) * kLsScale;
      m.w3[tid] = h16(W3[tid]);
    }
    if (tid == 0) m.b3 = h16(W3[kLsHid]);
  }
  if (blockIdx.x == 0 && tid == 0) A.counts[1] = 0;  // the touched list of this stage is counted after this kernel
  __syncthreads();
  double *su = m.u[warp];
  __half *sx = reinterpret_cast<__half *>(m.x[warp][0]), *sh = reinterpret_cast<__half *>(m.h[warp][0]);
  const int el = 2 * c + (g & 1);  // this lane's element
  const int ngroups = 16 * A.ntiles, gstep = gridDim.x * kLsWarps;
  constexpr int FILL = (8 * NP + 31) / 32;  // values per lane
  float fh[FILL], fl[FILL];
  int64_t nslot = 0;
  int nne = 0;
  double nh = 0.0;
  auto load = [&](int gi) {
    const MTile tl = A.tiles[gi >> 4];
    const int e0 = (gi & 15) * 8;
    const int ne = max(0, min(8, tl.nelem - e0));
    const int64_t base = tl.node_base + (int64_t)e0 * NP;
#pragma unroll
    for (int q = 0; q < FILL; ++q) {
      const int x = lane + 32 * q;
      fh[q] = x < ne * NP ? A.uhi[base + x] : 0.f;
      fl[q] = x < ne * NP ? A.ulo[base + x] : 0.f;
    }
    nslot = tl.elem_slot + e0;
    nne = ne;
    nh = (g < 2 && el < ne) ? A.h_over_n[nslot + el] : 0.0;
  };
  const int g0 = blockIdx.x * kLsWarps + warp;
  if (g0 < ngroups) load(g0);
  for (int gi = g0; gi < ngroups; gi += gstep) {
    const int64_t slot = nslot + el;
    const int ne = nne;
    const double hh = nh;
    if (lane == 0 && gi + gstep >= ngroups) pdl_trigger();
#pragma unroll
    for (int q = 0; q < FILL; ++q) {
      const int x = lane + 32 * q, e = x / NP;
      if (x < 8 * NP) su[e * SU + x - e * NP] = (double)fh[q] + (double)fl[q];
    }
    __syncwarp();
    if (gi + gstep < ngroups) load(gi + gstep);
    if (ne == 0) {
      __syncwarp();
      continue;  // past the tile's last element (warp-uniform)
    }
    // modal coefficients uhat = Vinv u of the 8 elements on the FP64 tensor path (mma.sync m8n8k4)
    double uh[MT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) uh[mt][0] = uh[mt][1] = 0.0;
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const int j = 4 * kk + c;
      const double bv = j < NP ? su[g * SU + j] : 0.0;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) ls_dmma(uh[mt][0], uh[mt][1], m.vinv[(mt * KT + kk) * 32 + lane], bv);
    }
    // energies: this lane's rows of elements 2c and 2c + 1, one of the two passed on in the first exchange
    double tot[2] = {0.0, 0.0}, top[2] = {0.0, 0.0};
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        tot[h] = fma(uh[mt][h], uh[mt][h], tot[h]);
        if ((topmask >> mt) & 1u) top[h] = fma(uh[mt][h], uh[mt][h], top[h]);
      }
    const bool odd = g & 1;
    double et = (odd ? tot[1] : tot[0]) + __shfl_xor_sync(0xffffffffu, odd ? tot[0] : tot[1], 4);
    double en = (odd ? top[1] : top[0]) + __shfl_xor_sync(0xffffffffu, odd ? top[0] : top[1], 4);
#pragma unroll
    for (int x = 8; x <= 16; x <<= 1) {
      et += __shfl_xor_sync(0xffffffffu, et, x);
      en += __shfl_xor_sync(0xffffffffu, en, x);
    }
    double sig = 0.0;
    if (A.mode != 0 && et > 0.0 && !(en < A.ratio0 * et)) sig = ls_pp_sigma(log10(en / et), A.s0, A.kappa);
    if (A.mode >= 2) {
      const double inv = et > 0.0 ? 1.0 / sqrt(et) : 0.0, other = __shfl_xor_sync(0xffffffffu, inv, 4);
      const double iv[2] = {odd ? other : inv, odd ? inv : other};
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (8 * mt + g < NP) ls_put(sx + (2 * c + h) * 2 * SX + 8 * mt + g, 16 * SX, (float)(uh[mt][h] * iv[h]));
      __syncwarp();
      // the network on the 8 elements with tensor products (mma.sync m16n8k16, FP16 operands, FP32 sums): the weights
      // are FP16 and each input a pair of FP16 parts, so the products keep FP32-level rounding.  Rows are hidden units
      // (two 16-row m-tiles), columns the warp's elements.
      float o[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        o[mt][0] = o[mt][1] = m.b1[16 * mt + g];
        o[mt][2] = o[mt][3] = m.b1[16 * mt + g + 8];
      }
      ls_layer<K1>(m.w + lane, m.x[warp][0] + g * SX + c, 8 * SX, o);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int f = 0; f < 4; ++f)
          ls_put(sh + (2 * c + (f & 1)) * 2 * SH + 16 * mt + g + 8 * (f >> 1), 16 * SH, tanhf(o[mt][f] * (1.f / kLsScale)));
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        o[mt][0] = o[mt][1] = m.b2[16 * mt + g];
        o[mt][2] = o[mt][3] = m.b2[16 * mt + g + 8];
      }
      ls_layer<K2>(m.w + K1 * 2 * 32 + lane, m.h[warp][0] + g * SH + c, 8 * SH, o);
      // output unit: this lane's four units of elements 2c and 2c + 1, summed over the lanes of the same c
      float za = 0.f, zb = 0.f;
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) {
        const float wlo = m.w3[16 * mt + g], whi = m.w3[16 * mt + g + 8];
        za += wlo * tanhf(o[mt][0] * (1.f / kLsScale)) + whi * tanhf(o[mt][2] * (1.f / kLsScale));
        zb += wlo * tanhf(o[mt][1] * (1.f / kLsScale)) + whi * tanhf(o[mt][3] * (1.f / kLsScale));
      }
#pragma unroll
      for (int x = 4; x <= 16; x <<= 1) {
        za += __shfl_xor_sync(0xffffffffu, za, x);
        zb += __shfl_xor_sync(0xffffffffu, zb, x);
      }
      const float sg = 1.f / (1.f + expf(-((odd ? zb : za) + m.b3)));
      // inside the low-confidence band the PP activation stands
      if (!(sg > A.conf_lo && sg < A.conf_hi)) sig = (A.mode == 3 && sg <= A.conf_lo) ? 0.0 : (double)sg;
    }
    bool active = false;
    if (g < 2 && el < ne) {
      const double eps = A.eps0 * sig * hh;
      A.eps[slot] = eps;
      active = eps > 0.0;
      int a = -1;
      if (active) {
        a = atomicAdd(&A.counts[0], 1);
        A.alist[a] = (int32_t)slot;
        A.tflag[slot] = 1;
      }
      A.aslot[slot] = a;
    }
    // An active element's neighbours, one of its four lanes (g mod 2 = el mod 2) per face.  slot_of_value walks the
    // partitions; with the four walks one after the other in the element's first lane the pass takes, every element
    // active, 117 us at order 2, 32^3 x 6 in 32 partitions and 448 at order 1, 48^3 x 6 in 48, for 61 and 194 so (in
    // one partition 44 and 115, for 39 and 99 so).
    if ((__ballot_sync(0xffffffffu, active) >> (lane & 7)) & 1u) {
      int node;
      const int64_t ns = slot_of_value(A, (int64_t)(uint32_t)A.conn[slot * kMixedConnWords + (g >> 1)], NP, &node);
      if (ns >= 0) A.tflag[ns] = 1;
    }
    __syncwarp();  // the warp's rows are free for its next group
  }
}

// touched list and row of every slot (-1 elsewhere); the flags are cleared for the next stage
__global__ void ls_compact_kernel(const LsArgs A) {
  pdl_wait();
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < A.nslots; s += step) {
    if (threadIdx.x == 0 && s + step >= A.nslots) pdl_trigger();
    if (A.tflag[s]) {
      const int r = atomicAdd(&A.counts[1], 1);
      A.tlist[r] = (int32_t)s;
      A.vslot[s] = r;
      A.tflag[s] = 0;
    } else {
      A.vslot[s] = -1;
    }
  }
}

// Sparse passes: one block of MT warps per group of 8 listed elements (the n-tile of the FP64 tensor path,
// mma.sync m8n8k4).  The block stages the group in shared memory (per-element offsets, eps and metrics; nodal
// values; face terms: each thread's few face points with their loads issued together), then warp mt applies the
// element matrices to rows 8 mt .. 8 mt + 7, reading their fragments transposed through L1 (DT[j][i], LT[m][i]:
// the few tens of KB stay there); lane l's output row is 8 mt + l / 4, its elements 2 (l mod 4) and
// 2 (l mod 4) + 1.  The mixed stage requires straight-sided elements, so the metrics are constant over an
// element and are read once per element.
//
// The list pass and the gradient let the next kernel start with their last group, the divergence not before its end.
// Started at once, the waiting CTAs cost more than the launch gap that they hide as soon as the lists are long (order 4,
// every element active, 32^3 x 6: 1204 us a stage, 994 so; 48^3 x 6: 3550 and 3293); the stage kernel waiting under the
// divergence's last groups costs 6 % at order 3 (32^3 x 6: 691 us a stage, 651 so).  With empty lists it is all the same.
template <int N>
struct LsCfg {
  using O = Order<N>;
  static constexpr int NP = O::NP, NF = O::NF;
  static constexpr int MT = (NP + 7) / 8, KT = (NP + 3) / 4, KL = NF / 4;
  static constexpr int NPU = 4 * KT;  // padded node rows of a staged element
  static constexpr int THREADS = 32 * MT;
  static constexpr int QF = (8 * NF + THREADS - 1) / THREADS;  // face points per thread
  static_assert(NF % 4 == 0, "face points in whole k-steps");
};

// per-element data of a staged group
struct LsElem {
  int64_t ub, fb;   // value offsets of the element in the state and face arrays
  double geo[9];    // rx .. tz (constant over a straight-sided element)
  double eps;
  int ok, act;      // listed element; row in the active list (-1: not active)
};

template <int N>
__device__ __forceinline__ void ls_stage_elems(const LsArgs &A, const int32_t *list, int n, int gi, LsElem *se,
                                               bool with_geo) {
  using C = LsCfg<N>;
  constexpr int NP = C::NP, NF = C::NF;
  const int t = threadIdx.x;
  if (t < 8) {
    LsElem x{};
    x.act = -1;
    if (8 * gi + t < n) {
      const int64_t slot = list[8 * gi + t];
      const int p = part_of_slot(A, slot);
      const int64_t le = slot - A.slot_prefix[p];
      x.ub = A.uoff[p] + le * NP;
      x.fb = A.foff[p] + le * NF;
      const int64_t gb = A.goff[p] + le * NP;
      if (with_geo)
        for (int m = 0; m < 9; ++m) x.geo[m] = A.geo[m][gb];
      x.eps = A.eps[slot];
      x.act = A.aslot[slot];
      x.ok = 1;
    }
    se[t] = x;
  }
}

template <int N>
__global__ void __launch_bounds__(LsCfg<N>::THREADS) ls_grad_kernel(const LsArgs A) {
  using C = LsCfg<N>;
  constexpr int NP = C::NP, NF = C::NF, KT = C::KT, KL = C::KL, NPU = C::NPU, QF = C::QF;
  __shared__ double su[8 * NPU], sj[3 * 8 * NF];
  __shared__ LsElem se[8];
  const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 5;
  const int ar = lane >> 2, ac = lane & 3, r = 8 * mt + ar;
  pdl_wait();
  const int n = *reinterpret_cast<volatile const int *>(&A.counts[0]);
  const int ngroups = (n + 7) / 8;
  for (int gi = blockIdx.x; gi < ngroups; gi += gridDim.x) {
    if (tid == 0 && gi + (int)gridDim.x >= ngroups) pdl_trigger();
    ls_stage_elems<N>(A, A.alist, n, gi, se, true);
    __syncthreads();
    for (int x = tid; x < 8 * NPU; x += C::THREADS) {
      const int e = x / NPU, i = x - e * NPU;
      su[x] = (se[e].ok && i < NP) ? (double)A.uhi[se[e].ub + i] + (double)A.ulo[se[e].ub + i] : 0.0;
    }
    // this thread's face points: gather indices and face data, then the neighbour traces
    int32_t g[QF];
    double nd[QF][4];
    bool use[QF];
#pragma unroll
    for (int b = 0; b < QF; ++b) {
      const int x = tid + C::THREADS * b, e = min(x / NF, 7), m = x - e * NF;
      use[b] = x < 8 * NF && se[e].ok;
      g[b] = use[b] ? A.gmap[se[e].fb + m] : 0;
      // straight-sided elements: normals and Fscale are constant over a face (its first point's values)
      for (int d = 0; d < 4; ++d) nd[b][d] = use[b] ? A.face[d][se[e].fb + (m / (NF / 4)) * (NF / 4)] : 0.0;
    }
    float ph[QF], pl[QF];
#pragma unroll
    for (int b = 0; b < QF; ++b) {
      const bool in = use[b] && (uint64_t)(int64_t)g[b] < (uint64_t)A.n_u_values;
      if (use[b] && !in) {
        atomicExch(A.status, kStatusBadGather);
        g[b] = -1;  // rejected index: the interior trace stands
      }
      ph[b] = in ? A.uhi[g[b]] : 0.f;
      pl[b] = in ? A.ulo[g[b]] : 0.f;
    }
    __syncthreads();  // su complete
#pragma unroll
    for (int b = 0; b < QF; ++b) {
      const int x = tid + C::THREADS * b;
      if (x < 8 * NF) {
        const int e = x / NF, m = x - e * NF;
        double jump = 0.0;
        if (use[b]) {
          const double uM = su[e * NPU + A.fmask[m]];
          const double uP = g[b] < 0 ? uM : (double)ph[b] + (double)pl[b];
          jump = 0.5 * (uP - uM) * nd[b][3];
        }
        for (int d = 0; d < 3; ++d) sj[(d * 8 + e) * NF + m] = nd[b][d] * jump;
      }
    }
    __syncthreads();  // sj complete
    double cr[2] = {0.0, 0.0}, cs[2] = {0.0, 0.0}, ct[2] = {0.0, 0.0};
    double cl[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const int j = 4 * kk + ac;
      const bool in = r < NP && j < NP;
      const double bv = su[ar * NPU + j];
      ls_dmma(cr[0], cr[1], in ? __ldg(A.Dr + j * NP + r) : 0.0, bv);
      ls_dmma(cs[0], cs[1], in ? __ldg(A.Ds + j * NP + r) : 0.0, bv);
      ls_dmma(ct[0], ct[1], in ? __ldg(A.Dt + j * NP + r) : 0.0, bv);
    }
#pragma unroll 5
    for (int kk = 0; kk < KL; ++kk) {
      const int m = 4 * kk + ac;
      const double al = r < NP ? __ldg(A.LIFT + m * NP + r) : 0.0;
#pragma unroll
      for (int d = 0; d < 3; ++d) ls_dmma(cl[d][0], cl[d][1], al, sj[(d * 8 + ar) * NF + m]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 2 * ac + h;
      if (r < NP && se[e].ok) {
        const LsElem &x = se[e];
        for (int d = 0; d < 3; ++d) {
          const double q = x.geo[d] * cr[h] + x.geo[3 + d] * cs[h] + x.geo[6 + d] * ct[h] + cl[d][h];
          A.eq[((int64_t)(8 * gi + e) * NP + r) * 3 + d] = x.eps * q;
        }
      }
    }
    __syncthreads();  // the staging buffers are free for the next group
  }
}

template <int N>
__global__ void __launch_bounds__(LsCfg<N>::THREADS) ls_div_kernel(const LsArgs A) {
  using C = LsCfg<N>;
  constexpr int NP = C::NP, NF = C::NF, KT = C::KT, KL = C::KL, NPU = C::NPU, QF = C::QF;
  __shared__ double sq[3 * 8 * NPU], sf[8 * NF];
  __shared__ LsElem se[8];
  const int tid = threadIdx.x, lane = tid & 31, mt = tid >> 5;
  const int ar = lane >> 2, ac = lane & 3, r = 8 * mt + ar;
  pdl_wait();
  const int n = *reinterpret_cast<volatile const int *>(&A.counts[1]);
  if (blockIdx.x == 0 && tid == 0) A.counts[0] = 0;  // the next stage's sensor pass counts from zero
  const int ngroups = (n + 7) / 8;
  for (int gi = blockIdx.x; gi < ngroups; gi += gridDim.x) {
    ls_stage_elems<N>(A, A.tlist, n, gi, se, true);
    __syncthreads();
    // the group's eps q_d, and this thread's face points: gather indices and face data
    for (int x = tid; x < 3 * 8 * NPU; x += C::THREADS) {  // node-major reads: a node's 3 values are adjacent
      const int e = x / (3 * NPU), y = x - e * 3 * NPU, i = y / 3, d = y - 3 * i;
      const int ae = se[e].act;
      sq[(d * 8 + e) * NPU + i] = (ae >= 0 && i < NP) ? A.eq[((int64_t)ae * NP + i) * 3 + d] : 0.0;
    }
    int32_t g[QF];
    double nd[QF][4];
    bool use[QF];
#pragma unroll
    for (int b = 0; b < QF; ++b) {
      const int x = tid + C::THREADS * b, e = min(x / NF, 7), m = x - e * NF;
      use[b] = x < 8 * NF && se[e].ok;
      g[b] = use[b] ? A.gmap[se[e].fb + m] : 0;
      // straight-sided elements: normals and Fscale are constant over a face (its first point's values)
      for (int d = 0; d < 4; ++d) nd[b][d] = use[b] ? A.face[d][se[e].fb + (m / (NF / 4)) * (NF / 4)] : 0.0;
    }
    // the neighbours' rows in the active list, then their eps q
    int an[QF], node[QF];
#pragma unroll
    for (int b = 0; b < QF; ++b) {
      an[b] = -1;
      node[b] = 0;
      if (use[b]) {
        const int64_t ns =
            ((uint64_t)(int64_t)g[b] < (uint64_t)A.n_u_values) ? slot_of_value(A, g[b], NP, &node[b]) : -1;
        if (ns >= 0)
          an[b] = A.aslot[ns];
        else
          atomicExch(A.status, kStatusBadGather);
      }
    }
    double ePq[QF][3];
#pragma unroll
    for (int b = 0; b < QF; ++b)
#pragma unroll
      for (int d = 0; d < 3; ++d) ePq[b][d] = an[b] >= 0 ? A.eq[((int64_t)an[b] * NP + node[b]) * 3 + d] : 0.0;
    __syncthreads();  // sq complete
#pragma unroll
    for (int b = 0; b < QF; ++b) {
      const int x = tid + C::THREADS * b;
      if (x < 8 * NF) {
        const int e = x / NF, m = x - e * NF;
        double flux = 0.0;
        if (use[b]) {
          const int jM = A.fmask[m];
          double v = 0.0;
          for (int d = 0; d < 3; ++d) v += nd[b][d] * (ePq[b][d] - sq[(d * 8 + e) * NPU + jM]);
          flux = 0.5 * nd[b][3] * v;
        }
        sf[e * NF + m] = flux;
      }
    }
    __syncthreads();  // every surface flux formed from sq
    // div(eps q) = sum_k D_k a_k with a_k = sum_d (d xi_k / d x_d) eps q_d (metrics constant over the element);
    // a_k replaces eps q_d in place, each thread owning whole nodes
    bool any_active = false;
    for (int e = 0; e < 8; ++e) any_active |= se[e].act >= 0;
    if (any_active) {
      for (int y = tid; y < 8 * NPU; y += C::THREADS) {
        const int e = y / NPU;
        if (se[e].act >= 0) {
          const double q0 = sq[y], q1 = sq[8 * NPU + y], q2 = sq[16 * NPU + y];
#pragma unroll
          for (int k = 0; k < 3; ++k)
            sq[k * 8 * NPU + y] = se[e].geo[3 * k] * q0 + se[e].geo[3 * k + 1] * q1 + se[e].geo[3 * k + 2] * q2;
        }
      }
      __syncthreads();
    }
    double c[3][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}}, cl[2] = {0.0, 0.0};
    if (any_active) {
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        const int j = 4 * kk + ac;
        const bool in = r < NP && j < NP;
        ls_dmma(c[0][0], c[0][1], in ? __ldg(A.Dr + j * NP + r) : 0.0, sq[ar * NPU + j]);
        ls_dmma(c[1][0], c[1][1], in ? __ldg(A.Ds + j * NP + r) : 0.0, sq[(8 + ar) * NPU + j]);
        ls_dmma(c[2][0], c[2][1], in ? __ldg(A.Dt + j * NP + r) : 0.0, sq[(16 + ar) * NPU + j]);
      }
    }
#pragma unroll 5
    for (int kk = 0; kk < KL; ++kk) {
      const int m = 4 * kk + ac;
      ls_dmma(cl[0], cl[1], r < NP ? __ldg(A.LIFT + m * NP + r) : 0.0, sf[ar * NF + m]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int e = 2 * ac + h;
      if (r < NP && se[e].ok) A.visc[(int64_t)(8 * gi + e) * NP + r] = (c[0][h] + c[1][h] + c[2][h]) + cl[h];
    }
    __syncthreads();  // the staging buffers are free for the next group
  }
}

template <int N>
void ls_attrs() {
  static bool done[64] = {};
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  if (dev >= 0 && dev < 64 && done[dev]) return;
  cuda_check(cudaFuncSetAttribute(ls_sensor_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(LsSensorSmem<N>)),
             "ls_sensor smem");
  if (dev >= 0 && dev < 64) done[dev] = true;
}

template <int N>
void launch_ls_n(const LsArgs &A, int num_sms, cudaStream_t st) {
  ls_attrs<N>();
  const int gs = std::max(1, std::min(2 * A.ntiles, num_sms * 3));
  launch_pdl(ls_sensor_kernel<N>, gs, 32 * kLsWarps, sizeof(LsSensorSmem<N>), st, A);
  launch_pdl(ls_compact_kernel, num_sms * 4, 256, 0, st, A);
  launch_pdl(ls_grad_kernel<N>, num_sms * 8, LsCfg<N>::THREADS, 0, st, A);
  launch_pdl(ls_div_kernel<N>, num_sms * 8, LsCfg<N>::THREADS, 0, st, A);
}

}  // namespace

bool ls_supported(int N) { return N >= 1 && N <= 4; }

void prepare_ls(int N) {
  switch (N) {
    case 1: ls_attrs<1>(); break;
    case 2: ls_attrs<2>(); break;
    case 3: ls_attrs<3>(); break;
    case 4: ls_attrs<4>(); break;
    default: break;
  }
}

void launch_ls(int N, const LsArgs &A, int num_sms, cudaStream_t st) {
  switch (N) {
    case 1: launch_ls_n<1>(A, num_sms, st); break;
    case 2: launch_ls_n<2>(A, num_sms, st); break;
    case 3: launch_ls_n<3>(A, num_sms, st); break;
    case 4: launch_ls_n<4>(A, num_sms, st); break;
    default: throw Error(DGK_ERR_UNSUPPORTED, "learned-sensor viscosity: orders 1..4");
  }
}

}  // namespace dgk
