// Artificial-viscosity stage with a modal shock sensor, and the sensor's small MLP (training and inference).
//
// Sensor (Persson & Peraire): per element the modal coefficients uhat = Vinv u (orthonormal simplex modes,
// order i, j, k), S = log10(energy of the modes of total degree N / total energy), activation
// sigma = 0 below s0 - kappa, 1 above s0 + kappa, (1 + sin(pi (S - s0) / (2 kappa))) / 2 between.  Learned
// sensor: sigma = MLP(uhat / |uhat|), a 35 -> 32 -> 32 -> 1 network (tanh, tanh, sigmoid) with FP16 weights and
// FP32 sums; where its output lies inside the low-confidence band (lo, hi) the element falls back to the PP
// activation.  Viscosity eps_e = eps0 sigma_e h_e / N, h_e = 2 / max Fscale over the element's face points.
//
// Viscous term (BR1 with central fluxes): q_d = D_d u + LIFT (Fscale n_d (uP - uM) / 2), d = x, y, z, then
// rhs += eps_e sum_d D_d q_d + LIFT (Fscale 1/2 sum_d n_d (epsP qP_d - epsM qM_d)), added to the
// Lax-Friedrichs right-hand side of the plain stage; the LSERK4 update follows in the same kernel.
//
// Three kernels per stage: av_sensor (eps per node), av_flux<GRAD> (q) and av_flux<RHS> (LF + viscous RHS + update).
// All products run on the FP64 tensor path (mma.sync m8n8k4) in groups of 8 elements.
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdint>

#include "dg_kernels.cuh"
#include "launch.cuh"
#include "tma.cuh"

namespace dgk {

namespace {

constexpr int kHid = 32;

__host__ __device__ constexpr int mlp_params(int nin) { return kHid * nin + kHid + kHid * kHid + kHid + kHid + 1; }

template <int N>
struct AvCfg {
  using O = Order<N>;
  static constexpr int NP = O::NP, NFP = O::NFP, NF = O::NF, NFS = frag_stride(NF);
  static constexpr int TE = N == 1 ? 32 : N == 2 ? 16 : 8;  // elements per tile: about 100 KB of ring for two CTAs per SM
  static constexpr int MT = (NP + 7) / 8, KT = (NP + 3) / 4, KL = NF / 4, NT = TE / 8;
};

__device__ __forceinline__ void av_dmma(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ double pp_sigma(double S, double s0, double kappa) {
  if (!(S >= s0 - kappa)) return 0.0;
  if (S > s0 + kappa) return 1.0;
  return 0.5 * (1.0 + sin(3.141592653589793 * (S - s0) / (2.0 * kappa)));
}

// ---- sensor pass: eps per node from the modal coefficients ----
//
// A warp takes 8 elements at a time: Vinv u as 8-row m-tiles on the FP64 tensor path, the energies by 4 lanes per
// element, the network (mode 2) with a hidden unit per lane and the 8 elements as independent sums.  The state of the
// warp's next group is loaded while the current one is computed.  24 us at order 4 and
// 82,944 elements with the Persson-Peraire sensor (0.93 TB/s of eps and u; bound by the FP64 chains of a warp).
constexpr int kSensorWarps = 8;

template <int N>
struct SensorSmem {
  static constexpr int NP = Order<N>::NP, NPS = Order<N>::NPS;
  double vinv[NP * NP];
  double uh[kSensorWarps][8 * NPS];
  float x[kSensorWarps][8 * NP], h1[kSensorWarps][8 * kHid], h2[kSensorWarps][8 * kHid];
  __half w[(mlp_params(NP) + 7) & ~7];
  int top[NP];
};

template <int N>
__global__ void __launch_bounds__(32 * kSensorWarps) av_sensor_kernel(const AvArgs A) {
  using C = AvCfg<N>;
  using S = SensorSmem<N>;
  constexpr int NP = C::NP, NPS = S::NPS, MT = C::MT, KT = C::KT, GPT = C::TE / 8;  // groups per tile
  constexpr int FILL = (8 * NP + 31) / 32;
  extern __shared__ __align__(16) unsigned char sm[];
  S &m = *reinterpret_cast<S *>(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int x = tid; x < NP * NP; x += blockDim.x) m.vinv[x] = A.Vinv[x];
  for (int x = tid; x < NP; x += blockDim.x) m.top[x] = A.top[x];
  pdl_wait();
  if (A.mode == 2)
    for (int x = tid; x < mlp_params(NP); x += blockDim.x) m.w[x] = __ushort_as_half(A.mlp16[x]);
  __syncthreads();
  double *uh = m.uh[warp];
  float *x = m.x[warp], *h1 = m.h1[warp], *h2 = m.h2[warp];
  const int ngroups = A.ntiles * GPT, gstep = gridDim.x * kSensorWarps;
  double v[FILL];
  AvTile tl{};
  int ne = 0;
  auto load = [&](int g) {
    tl = A.tiles[g / GPT];
    const int e0 = 8 * (g % GPT);
    ne = max(0, min(8, tl.nelem - e0));
    tl.node_base += (int64_t)e0 * NP;
    tl.elem_base += e0;
    tl.e1_base += e0;
    tl.feat_base += (int64_t)e0 * NP;
#pragma unroll
    for (int q = 0; q < FILL; ++q) v[q] = lane + 32 * q < ne * NP ? A.u[tl.node_base + lane + 32 * q] : 0.0;
  };
  const int g0 = blockIdx.x * kSensorWarps + warp;
  if (g0 < ngroups) load(g0);
  for (int g = g0; g < ngroups; g += gstep) {
    const AvTile cur = tl;
    const int cne = ne;
    if (lane == 0 && g + gstep >= ngroups) pdl_trigger();
#pragma unroll
    for (int q = 0; q < FILL; ++q) {
      const int i = lane + 32 * q, e = i / NP;
      if (i < 8 * NP) uh[e * NPS + i - e * NP] = v[q];
    }
    __syncwarp();
    if (g + gstep < ngroups) load(g + gstep);
    if (cne == 0) {
      __syncwarp();
      continue;  // past the tile's last element (warp-uniform)
    }
    {
      const int ar = lane >> 2, ac = lane & 3;
      double c[MT][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) c[mt][0] = c[mt][1] = 0.0;
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        const int j = 4 * kk + ac;
        const double bv = j < NP ? uh[ar * NPS + j] : 0.0;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int r = 8 * mt + ar;
          av_dmma(c[mt][0], c[mt][1], (r < NP && j < NP) ? m.vinv[r * NP + j] : 0.0, bv);
        }
      }
      __syncwarp();  // every lane's reads of the nodal values are done
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (8 * mt + ar < NP) uh[(2 * ac + h) * NPS + 8 * mt + ar] = c[mt][h];
      __syncwarp();
    }
    const int e = lane >> 2, t = lane & 3;  // 4 lanes per element
    const bool mine = e < cne;
    double tot = 0.0, hi = 0.0;
    for (int j = t; j < NP; j += 4) {
      const double w = uh[e * NPS + j];
      tot = fma(w, w, tot);
      if (m.top[j]) hi = fma(w, w, hi);
    }
    tot += __shfl_xor_sync(0xffffffffu, tot, 1);
    tot += __shfl_xor_sync(0xffffffffu, tot, 2);
    hi += __shfl_xor_sync(0xffffffffu, hi, 1);
    hi += __shfl_xor_sync(0xffffffffu, hi, 2);
    const double S = tot > 0.0 ? log10(hi / tot) : -INFINITY;
    const double pp = pp_sigma(S, A.s0, A.kappa);
    double sig = A.mode == 0 ? 0.0 : pp;  // sensor off: no viscosity
    if (mine && t == 0) {
      if (A.S_out) A.S_out[cur.e1_base + e] = (float)S;
      if (A.sig_out) A.sig_out[cur.e1_base + e] = (float)pp;
    }
    if (A.mode == 2 || A.feat_out) {  // unit-norm modal coefficients
      const double inv = tot > 0.0 ? 1.0 / sqrt(tot) : 0.0;
      for (int j = t; j < NP; j += 4) {
        const float f = (float)(uh[e * NPS + j] * inv);
        x[e * NP + j] = f;
        if (mine && A.feat_out) A.feat_out[cur.feat_base + (int64_t)e * NP + j] = f;
      }
      __syncwarp();
    }
    if (A.mode == 2) {
      // FP16 weights, FP32 sums in two chains per unit (lane) and element
      const __half *W1 = m.w, *b1 = W1 + kHid * NP, *W2 = b1 + kHid, *b2 = W2 + kHid * kHid, *w3 = b2 + kHid,
                   *b3 = w3 + kHid;
      float s0[8], s1[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        s0[k] = __half2float(b1[lane]);
        s1[k] = 0.f;
      }
#pragma unroll 1
      for (int j = 0; j + 1 < NP; j += 2) {
        const float wa = __half2float(W1[lane * NP + j]), wb = __half2float(W1[lane * NP + j + 1]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          s0[k] = fmaf(wa, x[k * NP + j], s0[k]);
          s1[k] = fmaf(wb, x[k * NP + j + 1], s1[k]);
        }
      }
      if (NP & 1) {
        const float wa = __half2float(W1[lane * NP + NP - 1]);
#pragma unroll
        for (int k = 0; k < 8; ++k) s0[k] = fmaf(wa, x[k * NP + NP - 1], s0[k]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) h1[k * kHid + lane] = tanhf(s0[k] + s1[k]);
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        s0[k] = __half2float(b2[lane]);
        s1[k] = 0.f;
      }
#pragma unroll 2
      for (int j = 0; j < kHid; j += 2) {
        const float wa = __half2float(W2[lane * kHid + j]), wb = __half2float(W2[lane * kHid + j + 1]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          s0[k] = fmaf(wa, h1[k * kHid + j], s0[k]);
          s1[k] = fmaf(wb, h1[k * kHid + j + 1], s1[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) h2[k * kHid + lane] = tanhf(s0[k] + s1[k]);
      __syncwarp();
      float z = __half2float(b3[0]);
      for (int j = 0; j < kHid; ++j) z = fmaf(__half2float(w3[j]), h2[e * kHid + j], z);
      const float sg = 1.f / (1.f + expf(-z));
      if (!(sg > A.conf_lo && sg < A.conf_hi)) {
        sig = sg;
      } else if (A.fallback_count && mine && t == 0) {
        atomicAdd(A.fallback_count, 1u);
      }
      if (A.mlp_out && mine && t == 0) A.mlp_out[cur.e1_base + e] = sg;
    }
    if (A.eps) {
      const double eps = mine ? A.eps0 * sig * A.h_over_n[cur.elem_base + e] : 0.0;
#pragma unroll
      for (int q = 0; q < FILL; ++q) {
        const int i = lane + 32 * q;
        const double w = __shfl_sync(0xffffffffu, eps, 4 * min(i / NP, 7));
        if (i < cne * NP) A.eps[cur.node_base + i] = w;
      }
    }
    __syncwarp();  // the warp's buffers are free for its next group
  }
}

// ---- BR1 gradient (RHS = false) and right-hand side with the LSERK4 update (RHS = true) ----
//
// Persistent CTAs, one consumer warp per (8-row m-tile, 8-element n-tile) with its A fragments of Dr, Ds, Dt and LIFT
// in registers.  A tile's node and face arrays stream through a two-slot ring of 1-D bulk copies; its neighbour values
// are gathered straight into the registers of the threads that form the face terms, one tile ahead (their gather
// indices two tiles ahead), so a tile waits for one memory round trip at most.  A bulk copy starts on 16 bytes: a
// tile may start on an odd value (odd Np and an odd element count before it), and is then copied from the value before.
// Two barriers per tile: the face terms are complete; the slot is free.
// Order 4, 82,944 elements: gradient 129 us (505 MB, 3.9 TB/s), right-hand side 126 us (598 MB, 4.7 TB/s; eps = 0), a
// stage 270 us with the sensor.  With one thread per node, the matrices in shared memory (a load per FMA) and the
// tile's loads, products and stores one after the other, the sensor and gradient took 719 us and the right-hand side 366.
// Bound by HBM and by the latency within a tile: two CTAs (98 KB of ring each) share an SM at order 4.
template <int N, bool RHS>
struct FluxCfg : AvCfg<N> {
  using C = AvCfg<N>;
  static constexpr int THREADS = 32 * C::MT * C::NT;
  static constexpr int NA = RHS ? 14 : 10;  // node arrays: u, 9 metrics; and q (3), resu
  static constexpr int F = RHS ? 1 : 3;     // face-term fields
  static constexpr int G = RHS ? 5 : 1;     // gathered values per face point: u; and eps, q (3)
  static constexpr uint32_t NODE_B = C::TE * C::NP * 8 + 16, FACE_B = C::TE * C::NF * 8 + 16;
  static constexpr uint32_t STAGE_B = NA * NODE_B + 4 * FACE_B;
  static constexpr size_t SMEM = 2 * (size_t)STAGE_B + F * C::TE * C::NFS * 8 + C::NF * 4 + 16;
  static constexpr int PER = (int)((227 * 1024) / (SMEM + 1024));  // CTAs that share an SM
  static constexpr int MINB = PER < 1 ? 1 : PER > 3 ? 3 : PER;
  static constexpr int NJ = (C::TE * C::NF + THREADS - 1) / THREADS;  // face points per thread
  static_assert(NODE_B % 16 == 0 && FACE_B % 16 == 0, "slots stay 16-byte aligned");
};

template <int N, bool RHS>
__device__ __forceinline__ void flux_issue(const AvArgs &A, const AvTile &tl, char *stage, uint64_t *bar) {
  using C = FluxCfg<N, RHS>;
  const int64_t nb = tl.node_base & ~(int64_t)1, fb = tl.face_base & ~(int64_t)1;
  const uint32_t nbytes = round16((uint32_t)((tl.nelem * C::NP + (int)(tl.node_base - nb)) * 8));
  const uint32_t fbytes = round16((uint32_t)((tl.nelem * C::NF + (int)(tl.face_base - fb)) * 8));
  mbar_expect_tx(bar, C::NA * nbytes + 4 * fbytes);
  bulk_g2s(stage, A.u + nb, nbytes, bar);
#pragma unroll
  for (int m = 0; m < 9; ++m) bulk_g2s(stage + (1 + m) * C::NODE_B, A.geo[m] + nb, nbytes, bar);
  if (RHS) {
#pragma unroll
    for (int d = 0; d < 3; ++d) bulk_g2s(stage + (10 + d) * C::NODE_B, A.q[d] + nb, nbytes, bar);
    bulk_g2s(stage + 13 * C::NODE_B, A.resu + nb, nbytes, bar);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) bulk_g2s(stage + C::NA * C::NODE_B + m * C::FACE_B, A.face[m] + fb, fbytes, bar);
}

template <int N, bool RHS>
__global__ void __launch_bounds__(FluxCfg<N, RHS>::THREADS, FluxCfg<N, RHS>::MINB) av_flux_kernel(const AvArgs A) {
  using C = FluxCfg<N, RHS>;
  constexpr int NP = C::NP, NF = C::NF, NFS = C::NFS, TE = C::TE, MT = C::MT, KT = C::KT, KL = C::KL, NJ = C::NJ;
  constexpr int THREADS = C::THREADS, NS = (int)(C::NODE_B / 8), FS = (int)(C::FACE_B / 8);  // array strides within a slot
  extern __shared__ __align__(128) unsigned char sm[];
  char *ring = reinterpret_cast<char *>(sm);
  double *sf = reinterpret_cast<double *>(ring + 2 * C::STAGE_B);  // [F][TE][NFS] face terms
  uint64_t *full = reinterpret_cast<uint64_t *>(sf + C::F * TE * NFS);
  int *sfm = reinterpret_cast<int *>(full + 2);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, step = gridDim.x;
  const int ntiles = A.ntiles;
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < NF; i += THREADS) sfm[i] = A.fmask[i];
  __syncthreads();
  const int mt = warp % MT, nt = warp / MT, ac = lane & 3, ar = lane >> 2;
  const int row = 8 * mt + ar;           // output node
  const int be = 8 * nt + ar;            // element of the B fragment
  const int ce = 8 * nt + 2 * ac;        // first of the two elements of the C fragment
  AvTile t0 = A.tiles[blockIdx.x], t1{};
  if (blockIdx.x + step < ntiles) t1 = A.tiles[blockIdx.x + step];
  double aD[3][KT], aL[KL];
#pragma unroll
  for (int kk = 0; kk < KT; ++kk) {
    const int j = 4 * kk + ac;
    const bool in = row < NP && j < NP;
    aD[0][kk] = in ? A.Dr[row * NP + j] : 0.0;
    aD[1][kk] = in ? A.Ds[row * NP + j] : 0.0;
    aD[2][kk] = in ? A.Dt[row * NP + j] : 0.0;
  }
#pragma unroll
  for (int kk = 0; kk < KL; ++kk) aL[kk] = row < NP ? A.LIFT[row * NF + 4 * kk + ac] : 0.0;
  pdl_wait();
  if (tid == 0) {
    flux_issue<N, RHS>(A, t0, ring, &full[0]);
    if (blockIdx.x + step < ntiles) flux_issue<N, RHS>(A, t1, ring + C::STAGE_B, &full[1]);
  }
  // this thread's face points: gather indices (two tiles ahead), gathered values (one tile ahead)
  int32_t idx[NJ];
  double gv[NJ][C::G], eM[NJ], eB = 0.0;
  uint32_t bad = 0;  // points whose index is out of range: the interior trace stands for the neighbour's
  auto load_idx = [&](const AvTile &tl) {
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int k = tid + j * THREADS;
      idx[j] = k < tl.nelem * NF ? __ldcs(A.gmap + tl.face_base + k) : 0;
    }
  };
  auto gather = [&](const AvTile &tl) {
    bad = 0;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int k = tid + j * THREADS;
      const bool in = k < tl.nelem * NF, ok = (uint64_t)(int64_t)idx[j] < (uint64_t)A.n_u_values;
      if (in && !ok) {
        bad |= 1u << j;
        atomicExch(A.status, kStatusBadGather);
      }
      gv[j][0] = in && ok ? A.u[idx[j]] : 0.0;
      if (RHS) {
        gv[j][1] = in && ok ? A.eps[idx[j]] : 0.0;
#pragma unroll
        for (int d = 0; d < 3; ++d) gv[j][2 + d] = in && ok ? A.q[d][idx[j]] : 0.0;
        eM[j] = in ? A.eps[tl.node_base + (k / NF) * NP] : 0.0;  // eps is constant over an element
      }
    }
    if (RHS) eB = be < tl.nelem ? A.eps[tl.node_base + be * NP] : 0.0;
  };
  load_idx(t0);
  gather(t0);
  if (blockIdx.x + step < ntiles) load_idx(t1);
  const double a = A.a, b = A.b, dt = A.dt;
  int k = 0;
  for (int t = blockIdx.x; t < ntiles; t += step, ++k) {
    const int s = k & 1;
    const bool has1 = t + step < ntiles, has2 = t + 2 * step < ntiles;
    if (tid == 0 && !has1) pdl_trigger();
    AvTile t2{};
    if (has2) t2 = A.tiles[t + 2 * step];
    const bool ready = mbar_wait_bounded(&full[s], (uint32_t)(k >> 1) & 1u, kSpinLimit);
    const int ne = t0.nelem, nfc = ne * NF;
    const char *stage = ring + s * C::STAGE_B;
    const double *su = reinterpret_cast<const double *>(stage) + (t0.node_base & 1);
    const double *sg = su + NS, *sq = su + 10 * NS, *sr = su + 13 * NS;
    const double *sfc = reinterpret_cast<const double *>(stage + C::NA * C::NODE_B) + (t0.face_base & 1);
    // face terms of this thread's points
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int x = tid + j * THREADS;
      if (x < nfc) {
        const int e = x / NF, m = x - e * NF, o = e * NP + sfm[m];
        const bool rejected = (bad >> j) & 1u;
        const double uM = su[o], uP = rejected ? uM : gv[j][0];
        const double nx = sfc[x], ny = sfc[FS + x], nz = sfc[2 * FS + x], fs = sfc[3 * FS + x];
        if (RHS) {
          const double ns = nx + ny + nz;
          const double fM = 0.5 * uM * uM * ns, fP = 0.5 * uP * uP * ns;
          const double lam = fmax(fabs(uM) * fabs(ns), fabs(uP) * fabs(ns));
          const double du = fM - (0.5 * (fM + fP) + 0.5 * lam * (uM - uP));
          const double eP = rejected ? eM[j] : gv[j][C::G > 1 ? 1 : 0];
          const double nv[3] = {nx, ny, nz};
          double vis = 0.0;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const double qM = sq[d * NS + o], qP = rejected ? qM : gv[j][C::G > 1 ? 2 + d : 0];
            vis += nv[d] * (eP * qP - eM[j] * qM);
          }
          sf[e * NFS + m] = fs * du + 0.5 * fs * vis;
        } else {
          const double jump = 0.5 * (uP - uM) * fs;
          sf[e * NFS + m] = nx * jump;
          sf[TE * NFS + e * NFS + m] = ny * jump;
          sf[2 * TE * NFS + e * NFS + m] = nz * jump;
        }
      }
    }
    const double eCur = eB;
    // in flight from here on: the next tile's neighbour values and the indices after them
    if (has1) gather(t1);
    if (has2) load_idx(t2);
    // derivatives at (row, ce), (row, ce + 1)
    double out[3][2];  // GRAD: q; RHS: out[0] = the volume terms
    {
      double c[3][2] = {};
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        const int j = 4 * kk + ac;
        const double bv = (j < NP && be < ne) ? su[be * NP + j] : 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) av_dmma(c[m][0], c[m][1], aD[m][kk], bv);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = (ce + h) * NP + row;
        const bool in = row < NP && ce + h < ne;
        double g[3] = {};
#pragma unroll
        for (int d = 0; d < 3; ++d)
          if (in) g[d] = sg[d * NS + o] * c[0][h] + sg[(3 + d) * NS + o] * c[1][h] + sg[(6 + d) * NS + o] * c[2][h];
        if (RHS) {
          out[0][h] = in ? -su[o] * (g[0] + g[1] + g[2]) : 0.0;
        } else {
#pragma unroll
          for (int d = 0; d < 3; ++d) out[d][h] = g[d];
        }
      }
    }
    if (RHS) {
      // eps div q where an element of the n-tile has viscosity
      if (__any_sync(0xffffffffu, eCur != 0.0)) {
        double div[2] = {};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double c[3][2] = {};
#pragma unroll
          for (int kk = 0; kk < KT; ++kk) {
            const int j = 4 * kk + ac;
            const double bv = (j < NP && be < ne) ? sq[d * NS + be * NP + j] : 0.0;
#pragma unroll
            for (int m = 0; m < 3; ++m) av_dmma(c[m][0], c[m][1], aD[m][kk], bv);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int o = (ce + h) * NP + row;
            if (row < NP && ce + h < ne)
              div[h] += sg[d * NS + o] * c[0][h] + sg[(3 + d) * NS + o] * c[1][h] + sg[(6 + d) * NS + o] * c[2][h];
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const double e = __shfl_sync(0xffffffffu, eCur, 4 * (2 * ac + h));  // element ce + h
          if (e != 0.0) out[0][h] += e * div[h];
        }
      }
    }
    if (!__syncthreads_and(ready)) {  // face terms complete; a wait that gave up ends every thread here
      if (tid == 0) atomicExch(A.status, kStatusTimeoutCode);
      mbar_wait_bounded(&full[s], (uint32_t)(k >> 1) & 1u, kSpinLimit);  // copies in flight land before the CTA goes
      if (has1) mbar_wait_bounded(&full[s ^ 1], (uint32_t)((k + 1) >> 1) & 1u, kSpinLimit);
      return;
    }
    // LIFT times the face terms
    {
      double c[3][2] = {};  // GRAD: the three directions; RHS: three chains of one sum
#pragma unroll
      for (int kk = 0; kk < KL; ++kk) {
        if (RHS) {
          av_dmma(c[kk % 3][0], c[kk % 3][1], aL[kk], be < ne ? sf[be * NFS + 4 * kk + ac] : 0.0);
        } else {
#pragma unroll
          for (int d = 0; d < 3; ++d)
            av_dmma(c[d][0], c[d][1], aL[kk], be < ne ? sf[(d * TE + be) * NFS + 4 * kk + ac] : 0.0);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = (ce + h) * NP + row;
        if (row < NP && ce + h < ne) {
          if (RHS) {
            const double rhs = out[0][h] + (c[0][h] + c[1][h] + c[2][h]);
            const double r = a * sr[o] + dt * rhs;
            __stcs(A.resu + t0.node_base + o, r);
            __stcs(A.u_out + t0.node_base + o, su[o] + b * r);
          } else {
#pragma unroll
            for (int d = 0; d < 3; ++d) A.q[d][t0.node_base + o] = out[d][h] + c[d][h];
          }
        }
      }
    }
    __syncthreads();  // every read of slot s and of the face terms is done
    if (tid == 0 && has2) {
      fence_async_smem();
      flux_issue<N, RHS>(A, t2, ring + s * C::STAGE_B, &full[s]);
    }
    t0 = t1;
    t1 = t2;
  }
}

template <int N>
void launch_av_n(const AvArgs &A, int num_sms, cudaStream_t st, LaunchInfo (&info)[3]) {
  const size_t s0 = sizeof(SensorSmem<N>);
  const int ps = info[0].per_sm = resident_ctas(av_sensor_kernel<N>, 32 * kSensorWarps, s0, &info[0]);
  const int groups = A.ntiles * (AvCfg<N>::TE / 8);
  const int gs = std::max(1, std::min((groups + kSensorWarps - 1) / kSensorWarps, ps * num_sms));
  launch_pdl(av_sensor_kernel<N>, gs, 32 * kSensorWarps, s0, st, A);
  if (A.prep_only) return;
  using Cg = FluxCfg<N, false>;
  using Cr = FluxCfg<N, true>;
  const int pg = info[1].per_sm = resident_ctas(av_flux_kernel<N, false>, Cg::THREADS, Cg::SMEM, &info[1]);
  launch_pdl(av_flux_kernel<N, false>, std::min(A.ntiles, pg * num_sms), Cg::THREADS, Cg::SMEM, st, A);
  const int pr = info[2].per_sm = resident_ctas(av_flux_kernel<N, true>, Cr::THREADS, Cr::SMEM, &info[2]);
  launch_pdl(av_flux_kernel<N, true>, std::min(A.ntiles, pr * num_sms), Cr::THREADS, Cr::SMEM, st, A);
}

// ---------------- MLP: forward, loss gradient (mean squared error), Adam, FP32 -> FP16 ----------------

template <int NIN>
__device__ __forceinline__ float mlp_fwd(const float *p, const float *x, float *h1, float *h2) {
  const float *W1 = p, *b1 = W1 + kHid * NIN, *W2 = b1 + kHid, *b2 = W2 + kHid * kHid, *w3 = b2 + kHid,
              *b3 = w3 + kHid;
#pragma unroll 4
  for (int o = 0; o < kHid; ++o) {
    float s = b1[o];
    for (int j = 0; j < NIN; ++j) s = fmaf(W1[o * NIN + j], x[j], s);
    h1[o] = tanhf(s);
  }
#pragma unroll 4
  for (int o = 0; o < kHid; ++o) {
    float s = b2[o];
    for (int j = 0; j < kHid; ++j) s = fmaf(W2[o * kHid + j], h1[j], s);
    h2[o] = tanhf(s);
  }
  float z = b3[0];
  for (int j = 0; j < kHid; ++j) z = fmaf(w3[j], h2[j], z);
  return 1.f / (1.f + expf(-z));
}

template <int NIN>
__global__ void mlp_forward_kernel(const float *p, const float *X, int64_t n, float *out) {
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
    float x[NIN], h1[kHid], h2[kHid];
    for (int j = 0; j < NIN; ++j) x[j] = X[s * NIN + j];
    out[s] = mlp_fwd<NIN>(p, x, h1, h2);
  }
}

// Gradient of mean((mlp(x) - y)^2) over n samples, added to `grad` (zeroed by the caller); `loss` receives the
// sum of squared errors / n.
//
// A block takes tiles of 64 samples through five small matrix products in shared memory (FP32 FMAs): both hidden
// layers, the back-propagated layer (W2^T d2) and the two weight gradients (d2 h1^T, d1 x^T).  Activations are
// stored [unit][sample], so a layer's thread (2 samples x 4 units) reads its samples as one float2 and its weights as
// one warp-uniform float4, and a gradient's thread reads 4 samples of a row at a time.  The gradients stay in
// registers over the block's tiles and reach memory as one atomic per parameter and block.
// 64 samples make 128 blocks of the trainer's batch of 8192: one wave.  The work (0.1 GFLOP at 35 inputs) is
// 1.5 us of FMAs; the kernel is bound by the latency of a tile's nine phases.  Measured (35 inputs, 8192 samples):
// a whole training step (zeroing, gradient, loss read-out, Adam) 4997 -> 50 us; the form before gave each sample to
// one thread, which added 2,273 shared-memory atomics per sample.
constexpr int kGradS = 64, kGradThreads = 256;  // samples per tile; 8 warps of 4 hidden units each

template <int NIN>
struct MlpGradSmem {
  static constexpr int LS = kGradS + 4;  // row of an activation: 16-byte aligned, rows 4 banks apart
  static constexpr int LW = kHid + 4;
  float x[NIN * LS], h1[kHid * LS], d[kHid * LS];           // d: d2, then d1
  float w1t[NIN * LW], w2t[kHid * LW], w2[kHid * LW];       // [in][out], [in][out], [out][in]
  float b1[kHid], b2[kHid], w3[kHid], zp[kHid / 4][kGradS], dz[kGradS], b3;
};

// acc[s][u] += sum_k w[k][u0 + u] a[k][s0 + s] for 2 samples and 4 units
template <int K>
__device__ __forceinline__ void mlp_tile_product(const float *w, int lw, const float *a, int la, float (&acc)[2][4]) {
#pragma unroll 8
  for (int k = 0; k < K; ++k) {
    const float2 v = *reinterpret_cast<const float2 *>(a + k * la);
    const float4 q = *reinterpret_cast<const float4 *>(w + k * lw);
    acc[0][0] = fmaf(q.x, v.x, acc[0][0]);
    acc[0][1] = fmaf(q.y, v.x, acc[0][1]);
    acc[0][2] = fmaf(q.z, v.x, acc[0][2]);
    acc[0][3] = fmaf(q.w, v.x, acc[0][3]);
    acc[1][0] = fmaf(q.x, v.y, acc[1][0]);
    acc[1][1] = fmaf(q.y, v.y, acc[1][1]);
    acc[1][2] = fmaf(q.z, v.y, acc[1][2]);
    acc[1][3] = fmaf(q.w, v.y, acc[1][3]);
  }
}

__device__ __forceinline__ float mlp_dot4(float4 a, float4 b, float s) {
  return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s))));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int m = 16; m; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

template <int NIN>
__global__ void __launch_bounds__(kGradThreads) mlp_grad_kernel(const float *p, const float *X, const float *y, int64_t n,
                                                                float *grad, float *loss) {
  using S = MlpGradSmem<NIN>;
  constexpr int LS = S::LS, LW = S::LW, KI = (NIN + 7) / 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  S &m = *reinterpret_cast<S *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int s0 = 2 * lane, u0 = 4 * warp;
  const float *W1 = p, *B1 = W1 + kHid * NIN, *W2 = B1 + kHid, *B2 = W2 + kHid * kHid, *W3 = B2 + kHid,
              *B3 = W3 + kHid;
  for (int i = tid; i < kHid * NIN; i += kGradThreads) m.w1t[(i % NIN) * LW + i / NIN] = W1[i];
  for (int i = tid; i < kHid * kHid; i += kGradThreads) {
    const float w = W2[i];
    m.w2t[(i % kHid) * LW + i / kHid] = w;
    m.w2[(i / kHid) * LW + i % kHid] = w;
  }
  if (tid < kHid) {
    m.b1[tid] = B1[tid];
    m.b2[tid] = B2[tid];
    m.w3[tid] = W3[tid];
  }
  if (tid == 0) m.b3 = B3[0];
  const float inv_n = 1.f / (float)n;
  float g1[KI] = {}, g2[4] = {}, gb1[4] = {}, gb2[4] = {}, gw3[4] = {}, gb3 = 0.f, ls = 0.f;
  const int64_t ntiles = (n + kGradS - 1) / kGradS;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t first = t * kGradS;
    const int ns = (int)min((int64_t)kGradS, n - first);
    __syncthreads();  // the previous tile's activations are read; first tile: the weights follow below
    for (int i = tid; i < kGradS * NIN; i += kGradThreads)
      m.x[(i % NIN) * LS + i / NIN] = i < ns * NIN ? X[first * NIN + i] : 0.f;
    const float yt = tid < ns ? y[first + tid] : 0.f;
    __syncthreads();
    float h1[2][4], h2[2][4], d2[2][4], d1[2][4];
    // hidden layers
#pragma unroll
    for (int u = 0; u < 4; ++u) h1[0][u] = h1[1][u] = m.b1[u0 + u];
    mlp_tile_product<NIN>(m.w1t + u0, LW, m.x + s0, LS, h1);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      h1[0][u] = tanhf(h1[0][u]);
      h1[1][u] = tanhf(h1[1][u]);
      *reinterpret_cast<float2 *>(m.h1 + (u0 + u) * LS + s0) = make_float2(h1[0][u], h1[1][u]);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) h2[0][u] = h2[1][u] = m.b2[u0 + u];
    mlp_tile_product<kHid>(m.w2t + u0, LW, m.h1 + s0, LS, h2);
    float z0 = 0.f, z1 = 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      h2[0][u] = tanhf(h2[0][u]);
      h2[1][u] = tanhf(h2[1][u]);
      z0 = fmaf(m.w3[u0 + u], h2[0][u], z0);
      z1 = fmaf(m.w3[u0 + u], h2[1][u], z1);
    }
    *reinterpret_cast<float2 *>(&m.zp[warp][s0]) = make_float2(z0, z1);
    __syncthreads();
    // output, its error and derivative: one thread per sample
    if (tid < kGradS) {
      float z = m.b3;
#pragma unroll
      for (int w = 0; w < kHid / 4; ++w) z += m.zp[w][tid];
      const float o = 1.f / (1.f + expf(-z));
      const float r = tid < ns ? o - yt : 0.f;
      const float dz = 2.f * r * o * (1.f - o) * inv_n;
      m.dz[tid] = dz;
      ls += r * r * inv_n;
      gb3 += dz;
    }
    __syncthreads();
    const float2 dz = *reinterpret_cast<const float2 *>(m.dz + s0);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float w = m.w3[u0 + u];
      d2[0][u] = dz.x * w * (1.f - h2[0][u] * h2[0][u]);
      d2[1][u] = dz.y * w * (1.f - h2[1][u] * h2[1][u]);
      gw3[u] += fmaf(dz.x, h2[0][u], dz.y * h2[1][u]);
      gb2[u] += d2[0][u] + d2[1][u];
      *reinterpret_cast<float2 *>(m.d + (u0 + u) * LS + s0) = make_float2(d2[0][u], d2[1][u]);
      d1[0][u] = d1[1][u] = 0.f;
    }
    __syncthreads();
    mlp_tile_product<kHid>(m.w2 + u0, LW, m.d + s0, LS, d1);
    {  // dW2: outputs (2 rows of d2) x (2 rows of h1) per thread
      const float *da = m.d + 2 * (tid >> 4) * LS, *ha = m.h1 + (tid & 15) * LS;
#pragma unroll 4
      for (int s = 0; s < kGradS; s += 4) {
        const float4 a0 = *reinterpret_cast<const float4 *>(da + s), a1 = *reinterpret_cast<const float4 *>(da + LS + s);
        const float4 c0 = *reinterpret_cast<const float4 *>(ha + s),
                     c1 = *reinterpret_cast<const float4 *>(ha + 16 * LS + s);
        g2[0] = mlp_dot4(a0, c0, g2[0]);
        g2[1] = mlp_dot4(a0, c1, g2[1]);
        g2[2] = mlp_dot4(a1, c0, g2[2]);
        g2[3] = mlp_dot4(a1, c1, g2[3]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      d1[0][u] *= 1.f - h1[0][u] * h1[0][u];
      d1[1][u] *= 1.f - h1[1][u] * h1[1][u];
      gb1[u] += d1[0][u] + d1[1][u];
    }
    __syncthreads();  // every read of d2 is done
#pragma unroll
    for (int u = 0; u < 4; ++u)
      *reinterpret_cast<float2 *>(m.d + (u0 + u) * LS + s0) = make_float2(d1[0][u], d1[1][u]);
    __syncthreads();
    {  // dW1: row tid / 8 of d1 times inputs tid mod 8 + 8 i
      const float *da = m.d + (tid >> 3) * LS, *xa = m.x + (tid & 7) * LS;
#pragma unroll 4
      for (int s = 0; s < kGradS; s += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(da + s);
#pragma unroll
        for (int i = 0; i < KI; ++i)
          if ((tid & 7) + 8 * i < NIN) g1[i] = mlp_dot4(a, *reinterpret_cast<const float4 *>(xa + 8 * i * LS + s), g1[i]);
      }
    }
  }
  float *G1 = grad, *Gb1 = G1 + kHid * NIN, *G2 = Gb1 + kHid, *Gb2 = G2 + kHid * kHid, *G3 = Gb2 + kHid,
        *Gb3 = G3 + kHid;
#pragma unroll
  for (int i = 0; i < KI; ++i)
    if ((tid & 7) + 8 * i < NIN) atomicAdd(&G1[(tid >> 3) * NIN + (tid & 7) + 8 * i], g1[i]);
#pragma unroll
  for (int i = 0; i < 4; ++i) atomicAdd(&G2[(2 * (tid >> 4) + (i >> 1)) * kHid + (tid & 15) + 16 * (i & 1)], g2[i]);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const float a = warp_sum(gb1[u]), b = warp_sum(gb2[u]), c = warp_sum(gw3[u]);
    if (lane == 0) {
      atomicAdd(&Gb1[u0 + u], a);
      atomicAdd(&Gb2[u0 + u], b);
      atomicAdd(&G3[u0 + u], c);
    }
  }
  if (warp < kGradS / 32) {
    const float a = warp_sum(gb3), b = warp_sum(ls);
    if (lane == 0) {
      atomicAdd(Gb3, a);
      atomicAdd(loss, b);
    }
  }
}

// zero the gradient and the loss before the gradient kernel
__global__ void mlp_zero_kernel(float *grad, int P, float *loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < P) grad[i] = 0.f;
  if (i == 0) *loss = 0.f;
}

__global__ void adam_kernel(float *p, const float *g, float *m, float *v, int64_t P, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < P; k += (int64_t)gridDim.x * blockDim.x) {
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.f - b1) * gk;
    const float vk = b2 * v[k] + (1.f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    p[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
  }
}

__global__ void to_half_kernel(const float *in, __half *out, int64_t n) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x)
    out[k] = __float2half_rn(in[k]);
}

// FP16-weight forward, the arithmetic of the sensor kernel: weights rounded to FP16, sums in FP32.
template <int NIN>
__global__ void mlp_forward16_kernel(const __half *p, const float *X, int64_t n, float *out) {
  constexpr int P = mlp_params(NIN);
  for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < n; s += (int64_t)gridDim.x * blockDim.x) {
    const __half *W1 = p, *b1 = W1 + kHid * NIN, *W2 = b1 + kHid, *b2 = W2 + kHid * kHid, *w3 = b2 + kHid,
                 *b3 = w3 + kHid;
    (void)P;
    float h1[kHid], h2[kHid];
    for (int o = 0; o < kHid; ++o) {
      float sum = __half2float(b1[o]);
      for (int j = 0; j < NIN; ++j) sum = fmaf(__half2float(W1[o * NIN + j]), X[s * NIN + j], sum);
      h1[o] = tanhf(sum);
    }
    for (int o = 0; o < kHid; ++o) {
      float sum = __half2float(b2[o]);
      for (int j = 0; j < kHid; ++j) sum = fmaf(__half2float(W2[o * kHid + j]), h1[j], sum);
      h2[o] = tanhf(sum);
    }
    float z = __half2float(b3[0]);
    for (int j = 0; j < kHid; ++j) z = fmaf(__half2float(w3[j]), h2[j], z);
    out[s] = 1.f / (1.f + expf(-z));
  }
}

}  // namespace

int mlp_param_count(int nin) { return mlp_params(nin); }

int av_tile_elems(int N) { return N == 1 ? AvCfg<1>::TE : N == 2 ? AvCfg<2>::TE : AvCfg<3>::TE; }

void launch_av(int N, const AvArgs &A, int num_sms, cudaStream_t st, LaunchInfo (&info)[3]) {
  switch (N) {
    case 1: launch_av_n<1>(A, num_sms, st, info); break;
    case 2: launch_av_n<2>(A, num_sms, st, info); break;
    case 3: launch_av_n<3>(A, num_sms, st, info); break;
    case 4: launch_av_n<4>(A, num_sms, st, info); break;
    case 5: launch_av_n<5>(A, num_sms, st, info); break;
    default: throw Error(DGK_ERR_UNSUPPORTED, "artificial-viscosity stage: orders 1..5");
  }
}

void launch_to_half(const float *in, void *out, int64_t n, cudaStream_t st) {
  to_half_kernel<<<std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4096)), 256, 0, st>>>(
      in, reinterpret_cast<__half *>(out), n);
  cuda_check(cudaGetLastError(), "to_half_kernel launch");
}

#define DGK_NIN_SWITCH(nin, CALL)                                                     \
  switch (nin) {                                                                      \
    case 4: CALL(4); break;                                                           \
    case 10: CALL(10); break;                                                         \
    case 20: CALL(20); break;                                                         \
    case 35: CALL(35); break;                                                         \
    case 56: CALL(56); break;                                                         \
    default: throw Error(DGK_ERR_UNSUPPORTED, "MLP input width must be Np of order 1..5"); \
  }

void launch_mlp_forward(const float *p, const float *X, int64_t n, int nin, float *out, int fp16, void *half_buf,
                        cudaStream_t st) {
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 127) / 128, 8192));
  if (fp16) {
    launch_to_half(p, half_buf, mlp_params(nin), st);
#define F16(NIN) mlp_forward16_kernel<NIN><<<blocks, 128, 0, st>>>(reinterpret_cast<const __half *>(half_buf), X, n, out)
    DGK_NIN_SWITCH(nin, F16)
#undef F16
  } else {
#define F32(NIN) mlp_forward_kernel<NIN><<<blocks, 128, 0, st>>>(p, X, n, out)
    DGK_NIN_SWITCH(nin, F32)
#undef F32
  }
  cuda_check(cudaGetLastError(), "mlp forward launch");
}

void launch_mlp_grad(const float *p, const float *X, const float *y, int64_t n, int nin, float *grad, float *loss,
                     cudaStream_t st) {
  const int P = mlp_params(nin);
  mlp_zero_kernel<<<(P + 255) / 256, 256, 0, st>>>(grad, P, loss);
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + kGradS - 1) / kGradS, 592));
#define G(NIN)                                                                                              \
  {                                                                                                         \
    cuda_check(cudaFuncSetAttribute(mlp_grad_kernel<NIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,      \
                                    (int)sizeof(MlpGradSmem<NIN>)),                                         \
               "mlp grad smem");                                                                            \
    mlp_grad_kernel<NIN><<<blocks, kGradThreads, sizeof(MlpGradSmem<NIN>), st>>>(p, X, y, n, grad, loss);   \
  }
  DGK_NIN_SWITCH(nin, G)
#undef G
  cuda_check(cudaGetLastError(), "mlp grad launch");
}

void launch_adam(float *p, const float *g, float *m, float *v, int64_t P, float lr, float b1, float b2, float eps,
                 int step, cudaStream_t st) {
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  adam_kernel<<<std::max<int64_t>(1, std::min<int64_t>((P + 255) / 256, 1024)), 256, 0, st>>>(p, g, m, v, P, lr, b1,
                                                                                                b2, eps, c1, c2);
  cuda_check(cudaGetLastError(), "adam launch");
}

}  // namespace dgk
