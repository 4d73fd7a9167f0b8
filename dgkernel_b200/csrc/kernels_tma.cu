// Fused strong-form Lax-Friedrichs RHS + LSERK4 stage, orders 1..5, TMA-pipelined for sm_100a with the element-local
// products on the FP64 tensor path.
//
// Persistent CTAs walk the tile list.  For every tile they stream, with 1-D bulk copies (cp.async.bulk, completion
// counted in bytes on an mbarrier), the tile's slice of the state, the residual, the nine per-node metrics and the four
// face arrays into a two-slot shared-memory ring: while tile t is computed, the copies of tile t+1 are in flight.  The
// neighbour traces are gathered through L2 by a producer warp.
//
// Every wait on an mbarrier is bounded: if a stage does not complete within the spin limit the kernel
// records kStatusTimeoutCode in the status word, waits (bounded) for the copies it issued, and returns.
#include <cstdint>
#include <type_traits>

#include "dg_kernels.cuh"
#include "launch.cuh"
#include "tma.cuh"
#include "kernels.hpp"
#include "runner.hpp"

namespace dgk {

// ------------------------------------------------------------------------------------------------
// The element-local products on the FP64 tensor path (mma.sync m8n8k4 .f64), arrays in FP64 or FP32 (ST).
//
// FP32 arrays move half the bytes and use the same FP64 products (FP32 operands are exact in FP64, and the sums are
// FP64's): 1.1 G FMAs a stage at order 4 and 32^3 x 6 are 62 us at the FP64 rate, under the 91 us of its bytes, where
// the FP32 cores need a shared-memory matrix entry per FMA.  Flux, metrics and update stay in FP32.  Their tiles hold two
// n-tiles per warp from order 3 on: the barriers and waits of a tile then serve 16 elements.
// Order 4, 32^3 x 6: 182 us a stage from 247 with the register-staged form on the FP32 cores.
//
// The products OUT = M * U of a tile are small GEMMs: M is NP x NP (Dr, Ds, Dt) or NP x NF (LIFT), U holds
// the TE element vectors of the tile as columns.  Warp w owns rows 8w..8w+7 (one m-tile) of every matrix
// and keeps its A fragments for all k-steps in registers for the whole persistent kernel; per tile it only
// loads B fragments (element values) from the shared-memory ring.  Fragment layouts of m8n8k4 .f64:
// A (8x4, row-major): lane l holds A[l>>2][l&3]; B (4x8, column-major): lane l holds B[l&3][l>>2];
// C/D (8x8): lane l holds C[l>>2][2(l&3)] and C[l>>2][2(l&3)+1].
// ------------------------------------------------------------------------------------------------
// elements per tile, n-tiles (8 elements) per consumer warp
template <int N, typename ST>
struct DmmaShape {
  static constexpr bool F32 = sizeof(ST) == 4;
  static constexpr int TE = N == 1 ? 32 : N == 2 || F32 ? 16 : 8;
  static constexpr int NW = N >= 3 && F32 ? 2 : 1;
};

// CP: compact FP64 form (per element: the kCompactGeo64 constant geometry values instead of the 9 metric and
// 4 face arrays; neighbour traces through the compact connectivity instead of the gather map)
template <int N, bool CP, typename T>
struct DmmaCfg {
  using O = Order<N>;
  static constexpr int NP = O::NP, NF = O::NF, NFS = frag_stride(NF);
  static constexpr int TE = DmmaShape<N, T>::TE, NW = DmmaShape<N, T>::NW;
  static constexpr int MT = (NP + 7) / 8;  // m-tiles (8 rows)
  static constexpr int KT = (NP + 3) / 4;  // k-steps of the derivative matrices
  static constexpr int KL = NF / 4;        // k-steps of LIFT (NF = 4 Nfp)
  static constexpr int NT = TE / 8;        // n-tiles (8 elements)
  static constexpr int CONS = 32 * MT * NT / NW;  // consumer threads: one warp per (m-tile, NW n-tiles)
  // Producer warps gathering neighbour traces.  The compact form's producer resolves a connectivity word and a table
  // entry per point, which at orders 1 and 2 takes longer than the tile's products: with two warps a stage takes 48 and
  // 133 us for 94 and 191 (40^3 x 6).  From order 3 on the products are the longer part, and a second one is slower.
  static constexpr int PW = CP && N <= 2 ? 2 : 1;
  static constexpr int THREADS = CONS + 32 * PW;
  // a bulk copy starts on 16 bytes; a tile that does not is copied from the 16 bytes that hold its start
  static constexpr int AV = 16 / sizeof(T);  // values per 16 bytes
  static constexpr uint32_t NODE_B = TE * NP * sizeof(T) + 16;
  static constexpr uint32_t FACE_B = TE * NF * sizeof(T) + 16;
  static constexpr int NS = NODE_B / sizeof(T), FS = FACE_B / sizeof(T);  // array strides within a slot
  static constexpr uint32_t GEOC_B = (uint32_t)TE * kCompactGeo64 * sizeof(double);
  // u, resu, then 9 metrics and 4 face arrays, or the compact geometry
  static constexpr uint32_t STAGE_B = CP ? 2 * NODE_B + GEOC_B : 11 * NODE_B + 4 * FACE_B;
  static constexpr uint32_t GBUF_B = TE * NF * sizeof(T);         // gathered uP of one tile
  // two gathered-uP buffers, two surface-flux buffers (a warp may start the next tile's flux while another
  // still reads this tile's in the LIFT product), the face-point mask
  static constexpr uint32_t WORK_B = 2 * GBUF_B + 2 * TE * NFS * sizeof(double) + NF * sizeof(int32_t);
  static constexpr int FTR = (NF / 4 + 15) & ~15;        // face-order table row: Nfp bytes rounded up to 16
  static constexpr uint32_t FTAB_B = CP ? 256 * FTR : 0;
  static constexpr size_t SMEM = 2 * (size_t)STAGE_B + WORK_B + 10 * sizeof(uint64_t) + FTAB_B;
  // Co-resident CTAs that the launch bounds plan for.  At order 5 the compact form holds two only with a few registers
  // spilled, which is still the faster (24^3 x 6: 178 us a stage, one CTA 242); the FP32 form runs one.
  static constexpr int MINB = (CP || N < 5) && 2 * SMEM <= 227 * 1024 ? 2 : 1;
  static constexpr int GJ = (TE * NF + 32 * PW - 1) / (32 * PW);  // gathers per producer lane and tile
  static_assert(NODE_B % 16 == 0 && FACE_B % 16 == 0 && GBUF_B % 16 == 0 && GEOC_B % 16 == 0,
                "smem slots must stay 16-byte aligned");
  static_assert(TE % 8 == 0 && NF % 4 == 0 && NT % NW == 0, "tile must be whole n-tiles");
};

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}


// Barrier among the consumer warps only (named barrier 1), and its AND-reduction form.
template <int CONS>
__device__ __forceinline__ void cons_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(CONS) : "memory");
}
template <int CONS>
__device__ __forceinline__ bool cons_sync_and(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred q, o;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.and.pred o, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, o;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p), "n"(CONS)
      : "memory");
  return r != 0;
}

// A tile's stage is filled in two parts with their own barriers: part A (the 9 metrics and 4 face arrays, read
// by the volume products and the flux) and part B (u and resu, read until the update).
template <int N, bool CP, typename T>
__device__ __forceinline__ void issue_tile_a(const RhsArgs<T> &A, const Tile &tl, int64_t slot, char *stage,
                                             uint64_t *bar) {
  using C = DmmaCfg<N, CP, T>;
  if (CP) {  // the compact geometry of the tile's element slots (slots are padded to whole tiles)
    mbar_expect_tx(bar, C::GEOC_B);
    bulk_g2s(stage + 2 * C::NODE_B, A.geoc + slot * kCompactGeo64, C::GEOC_B, bar);
    return;
  }
  const int ns = (int)(tl.node_base & (C::AV - 1)), fs = (int)(tl.face_base & (C::AV - 1));
  const uint32_t nb = round16((uint32_t)((tl.nelem * C::NP + ns) * sizeof(T)));
  const uint32_t fb = round16((uint32_t)((tl.nelem * C::NF + fs) * sizeof(T)));
  mbar_expect_tx(bar, 9 * nb + 4 * fb);
#pragma unroll
  for (int m = 0; m < 9; ++m) bulk_g2s(stage + (2 + m) * C::NODE_B, A.geo[m] + tl.node_base - ns, nb, bar);
#pragma unroll
  for (int m = 0; m < 4; ++m)
    bulk_g2s(stage + 11 * C::NODE_B + m * C::FACE_B, A.face[m] + tl.face_base - fs, fb, bar);
}

template <int N, bool CP, typename T>
__device__ __forceinline__ void issue_tile_b(const RhsArgs<T> &A, const Tile &tl, char *stage, uint64_t *bar,
                                             int rhs_only) {
  using C = DmmaCfg<N, CP, T>;
  const int ns = (int)(tl.node_base & (C::AV - 1));
  const uint32_t nb = round16((uint32_t)((tl.nelem * C::NP + ns) * sizeof(T)));
  mbar_expect_tx(bar, (rhs_only ? 1 : 2) * nb);
  bulk_g2s(stage, A.u_in + tl.node_base - ns, nb, bar);
  if (!rhs_only) bulk_g2s(stage + C::NODE_B, A.resu + tl.node_base - ns, nb, bar);
}

// Gather indices of one tile's face points for producer lane `lane` (points lane, lane + 32, ...), in two parts
// so the loads can be in flight a tile ahead: dmma_gather_load issues the loads (the gather map entry; in the
// compact form the neighbour's base and the face-order codes from the compact connectivity), and
// dmma_gather_finish adds the point's node from the face-order table (compact form only).
// Points past the tile's last element get 0 (never read).
template <int N, bool CP, typename T>
__device__ __forceinline__ void dmma_gather_load(const RhsArgs<T> &A, const Tile &tl, int64_t slot0, int lane,
                                                 int32_t (&src)[DmmaCfg<N, CP, T>::GJ],
                                                 uint32_t (&code)[DmmaCfg<N, CP, T>::GJ]) {
  using C = DmmaCfg<N, CP, T>;
  constexpr int NF = C::NF, GJ = C::GJ;
  const int nfc = tl.nelem * NF;
#pragma unroll
  for (int j = 0; j < GJ; ++j) {
    const int idx = lane + 32 * C::PW * j;
    src[j] = 0;
    code[j] = 0;
    if (idx < nfc) {
      if (CP) {
        const int e = idx / NF, f = (idx - e * NF) / (NF / 4);
        const int32_t *cn = A.conn + (slot0 + e) * kMixedConnWords;
        src[j] = cn[f];
        code[j] = (uint32_t)cn[4];
      } else {
        src[j] = __ldcs(A.gmap + tl.face_base + idx);
      }
    }
  }
}

template <int N, bool CP, typename T>
__device__ __forceinline__ void dmma_gather_finish(const RhsArgs<T> &A, const Tile &tl, const uint8_t *sft, int lane,
                                                   int32_t (&src)[DmmaCfg<N, CP, T>::GJ],
                                                   const uint32_t (&code)[DmmaCfg<N, CP, T>::GJ]) {
  if (!CP) return;
  using C = DmmaCfg<N, CP, T>;
  constexpr int NF = C::NF, GJ = C::GJ, NFP = NF / 4;
  const int nfc = tl.nelem * NF;
  const int ncd = min(A.ncodes, 256);
#pragma unroll
  for (int j = 0; j < GJ; ++j) {
    const int idx = lane + 32 * C::PW * j;
    if (idx < nfc) {  // the point's face-order code, then the point's node in the neighbour
      const int e = idx / NF, q = idx - e * NF, f = q / NFP, p = q - f * NFP;
      const int cd = min((int)((code[j] >> (8 * f)) & 0xffu), ncd - 1);
      src[j] += sft[cd * C::FTR + p];
    }
  }
}

// Warp-specialized CTA.  Producer warp: for tile k it reads the tile's gather map and the neighbour traces uP
// from global memory (one batch of loads per lane), writes them to gbuf[k & 1] and signals gready; it runs up
// to two tiles ahead, gated by gfree.  Consumer warps: wait for the TMA stage and gready, then
// (a) [Dr;Ds;Dt] * U on the tensor path with the metrics applied in the epilogue (volume terms stay in
// registers), (b) the Lax-Friedrichs flux of their face points, (c) LIFT * flux on the tensor path with the
// LSERK4 update in the epilogue, streamed to HBM.  One consumer barrier per tile, after the flux (it also
// AND-reduces the waits' outcome, so a timed-out wait ends every consumer there); the end of a tile is a
// counter instead: each consumer warp adds one when it has read the slot's u and resu, and the last one issues
// the slot's refill, so a warp goes on to the next tile without waiting for the others.  The flux buffer
// alternates with the slot: warps are at most one tile apart (the next barrier needs all of them).
template <int N, bool CP, typename T>
__global__ void __launch_bounds__(DmmaCfg<N, CP, T>::THREADS, DmmaCfg<N, CP, T>::MINB)
    rhs_stage_dmma_kernel(RhsArgs<T> A, int rhs_only) {
  using C = DmmaCfg<N, CP, T>;
  constexpr int NP = C::NP, NF = C::NF, NFS = C::NFS, TE = C::TE, CONS = C::CONS;
  constexpr int KT = C::KT, KL = C::KL, MT = C::MT, GJ = C::GJ, NW = C::NW, NS = C::NS, FS = C::FS;
  constexpr int LDD = pad_even(NP), LDL = pad_even(NF);
  constexpr int NJ = (TE * NF + CONS - 1) / CONS;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  char *ring = reinterpret_cast<char *>(smem_raw);
  T *gbuf = reinterpret_cast<T *>(ring + 2 * C::STAGE_B);                 // [2][TE*NF] gathered uP
  double *sf2 = reinterpret_cast<double *>(gbuf + 2 * TE * NF);             // [2][TE*NFS] surface flux of the tile
  int *sfm = reinterpret_cast<int *>(sf2 + 2 * TE * NFS);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sfm + NF);    // fullA[2], gready[2], gfree[2], fullB[2]
  uint64_t *full = bar, *gready = bar + 2, *gfree = bar + 4, *fullb = bar + 6;
  int *done = reinterpret_cast<int *>(bar + 8);          // [2] consumer warps done with the slot's u and resu
  uint8_t *sft = reinterpret_cast<uint8_t *>(bar + 10);  // compact form: face-order rows of C::FTR bytes
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x;
  if (tid == 0) {
    for (int i = 0; i < 8; ++i) mbar_init(&bar[i], i == 2 || i == 3 ? C::PW : 1);
    done[0] = done[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < NF; i += C::THREADS) sfm[i] = A.fmask[i];
  if (CP) {
    constexpr int NFP = NF / 4;
    for (int i = tid; i < min(A.ncodes, 256) * C::FTR; i += C::THREADS) {
      const int row = i / C::FTR, col = i - row * C::FTR;
      sft[i] = col < NFP ? A.ftab[row * NFP + col] : 0;
    }
  }
  __syncthreads();

  if (tid >= CONS) {
    const int plane = C::PW == 1 ? lane : tid - CONS;  // lane among the producer warps
    pdl_wait();
    // ---------------- producer warp: neighbour traces ----------------
    // Software-pipelined over the CTA's tiles: while the traces of tile t are gathered, the loads of tile t + G's
    // gather indices (from its descriptor, loaded one tile earlier) and of tile t + 2G's descriptor are in
    // flight, so a tile costs one dependent round trip to memory instead of three (64^3 x 6 order 4: the stage
    // went from 2.17 to 1.94 ms).
    Tile tl = A.tiles[blockIdx.x], tn = {};
    int64_t sl = CP ? A.tile_slot[blockIdx.x] : 0, sn = 0;
    if (blockIdx.x + G < A.ntiles) {
      tn = A.tiles[blockIdx.x + G];
      if (CP) sn = A.tile_slot[blockIdx.x + G];
    }
    // The compact form's index loads feed arithmetic (the face-order table) at once, so it is not pipelined: its
    // loads are issued after the wait for the tile's buffer (pipelined, the compact stage ran 5% slower).
    int32_t src[GJ];
    uint32_t code[GJ];
    if (!CP) dmma_gather_load<N, CP, T>(A, tl, sl, plane, src, code);
    int k = 0;
    for (int t = blockIdx.x; t < A.ntiles; t += G, ++k) {
      const int s = k & 1;
      if (k >= 2 && !mbar_wait_bounded(&gfree[s], ((k >> 1) - 1) & 1, kSpinLimit)) {
        if (lane == 0) atomicExch(A.status, kStatusTimeoutCode);
        return;  // consumers time out on gready and leave as well
      }
      if (CP) dmma_gather_load<N, CP, T>(A, tl, sl, plane, src, code);
      dmma_gather_finish<N, CP, T>(A, tl, sft, plane, src, code);
      const int nfc = tl.nelem * NF;
      T up[GJ];
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        const int idx = plane + 32 * C::PW * j;
        up[j] = T(0);
        if (idx < nfc) {
          if (src[j] >= 0 && (int64_t)src[j] < A.n_u_values) {
            up[j] = __ldcg(A.u_in + src[j]);
          } else {  // rejected index: report it and use the interior trace
            atomicExch(A.status, kStatusBadGather);
            const int e = idx / NF, q = idx - e * NF;
            up[j] = A.u_in[tl.node_base + e * NP + sfm[q]];
          }
        }
      }
      // in flight with the gathers: the next tile's indices and the descriptor after it
      Tile tnn = {};
      int64_t snn = 0;
      if (t + 2 * G < A.ntiles) {
        tnn = A.tiles[t + 2 * G];
        if (CP) snn = A.tile_slot[t + 2 * G];
      }
      if (!CP && t + G < A.ntiles) dmma_gather_load<N, CP, T>(A, tn, sn, plane, src, code);
      T *g = gbuf + s * TE * NF;
#pragma unroll
      for (int j = 0; j < GJ; ++j) {
        const int idx = plane + 32 * C::PW * j;
        if (idx < nfc) g[idx] = up[j];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&gready[s]);
      tl = tn;
      sl = sn;
      tn = tnn;
      sn = snn;
    }
    return;
  }

  // ---------------- consumer warps ----------------
  const int mt = warp % MT, nt = warp / MT;
  const int arow = mt * 8 + (lane >> 2);  // output row of this lane (A row, C row)
  const int acol = lane & 3;              // column within a k-step (A col, B row)
  const int be = nt * NW * 8 + (lane >> 2);  // element of this lane's B fragment (of the warp's first n-tile)
  const int ce = nt * NW * 8 + 2 * acol;     // first of the two elements of this lane's C fragment
  // A fragments of Dr, Ds, Dt and LIFT for this warp's m-tile, resident for the kernel's lifetime
  double aD[3][KT], aL[KL];
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const int j = 4 * kk + acol;
      aD[m][kk] = (arow < NP && j < NP) ? A.D64[(m * NP + arow) * LDD + j] : 0.0;
    }
#pragma unroll
  for (int kk = 0; kk < KL; ++kk) aL[kk] = arow < NP ? A.L64[arow * LDL + 4 * kk + acol] : 0.0;
  pdl_wait();
  if (tid == 0) {
    for (int j = 0; j < 2; ++j)
      if ((int)blockIdx.x + j * G < A.ntiles) {
        const Tile tj = A.tiles[blockIdx.x + j * G];
        issue_tile_a<N, CP, T>(A, tj, CP ? A.tile_slot[blockIdx.x + j * G] : 0, ring + j * C::STAGE_B, &full[j]);
        issue_tile_b<N, CP, T>(A, tj, ring + j * C::STAGE_B, &fullb[j], rhs_only);
      }
  }
  const T a = A.a, b = A.b, dt = A.dt;
  constexpr int CW = CONS / 32;  // consumer warps
  // tile descriptors in registers: this tile's and the next were loaded in earlier iterations; tile t + 2G's
  // (read by the refills mid-tile) is loaded at the top of the iteration, before the waits
  Tile tcur = A.tiles[blockIdx.x];
  Tile tnext = blockIdx.x + G < A.ntiles ? A.tiles[blockIdx.x + G] : Tile{};
  int k = 0;
  for (int t = blockIdx.x; t < A.ntiles; t += G, ++k) {
    const int s = k & 1;
    const uint32_t parity = (k >> 1) & 1;
    const bool has2 = t + 2 * G < A.ntiles;
    if (tid == 0 && t + G >= A.ntiles) pdl_trigger();
    Tile t2 = {};
    int64_t slot2 = 0;
    if (has2) {
      t2 = A.tiles[t + 2 * G];
      if (CP) slot2 = A.tile_slot[t + 2 * G];
    }
    // a wait that gives up leaves the slot unread: the tile is computed from whatever the slot holds (every
    // index stays inside the shared-memory buffers) and the barrier after the flux ends all consumers
    const bool ready = mbar_wait_bounded(&full[s], parity, kSpinLimit) &&
                       mbar_wait_bounded(&fullb[s], parity, kSpinLimit) &&
                       mbar_wait_bounded(&gready[s], parity, kSpinLimit);
    const Tile tl = tcur;
    const int ne = tl.nelem, nfc = ne * NF;
    const char *stage = ring + s * C::STAGE_B;
    const T *su = reinterpret_cast<const T *>(stage) + (tl.node_base & (C::AV - 1));
    const T *sr = su + NS;
    const T *sg = su + 2 * NS;  // per-node metrics
    const double *sgc = reinterpret_cast<const double *>(stage + 2 * C::NODE_B);  // compact form: per-element geometry
    const T *sfc = reinterpret_cast<const T *>(stage + 11 * C::NODE_B) + (tl.face_base & (C::AV - 1));
    const T *g = gbuf + s * TE * NF;
    double *sf = sf2 + s * TE * NFS;

    // (a) ur, us, ut on the tensor path; with one n-tile, two interleaved accumulator chains per matrix
    T vol[NW][2];
    {
      constexpr int CH = NW == 1 ? 2 : 1;
      double c[NW][3][CH][2];
#pragma unroll
      for (int n = 0; n < NW; ++n)
#pragma unroll
        for (int m = 0; m < 3; ++m)
#pragma unroll
          for (int h = 0; h < CH; ++h) c[n][m][h][0] = c[n][m][h][1] = 0.0;
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        const int j = 4 * kk + acol;
#pragma unroll
        for (int n = 0; n < NW; ++n) {
          double bv = (j < NP && be + 8 * n < ne) ? (double)su[(be + 8 * n) * NP + j] : 0.0;
          if (A.conservative) bv = 0.5 * bv * bv;
#pragma unroll
          for (int m = 0; m < 3; ++m) dmma(c[n][m][kk % CH][0], c[n][m][kk % CH][1], aD[m][kk], bv);
        }
      }
      // epilogue: metrics at (element, node) and the volume term of the reference's quasi-linear form
#pragma unroll
      for (int n = 0; n < NW; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = ce + 8 * n + h;
          vol[n][h] = T(0);
          if (arow < NP && e < ne) {
            const int o = e * NP + arow;
            const T ur = (T)(c[n][0][0][h] + (CH == 2 ? c[n][0][CH - 1][h] : 0.0));
            const T us = (T)(c[n][1][0][h] + (CH == 2 ? c[n][1][CH - 1][h] : 0.0));
            const T ut = (T)(c[n][2][0][h] + (CH == 2 ? c[n][2][CH - 1][h] : 0.0));
            T m9[9];
#pragma unroll
            for (int m = 0; m < 9; ++m) m9[m] = CP ? (T)sgc[e * kCompactGeo64 + m] : sg[m * NS + o];
            const T ux = m9[0] * ur + m9[3] * us + m9[6] * ut;
            const T uy = m9[1] * ur + m9[4] * us + m9[7] * ut;
            const T uz = m9[2] * ur + m9[5] * us + m9[8] * ut;
            vol[n][h] = A.conservative ? -(ux + uy + uz) : -su[o] * (ux + uy + uz);
          }
        }
    }
    // (b) Lax-Friedrichs flux of this thread's face points
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int idx = tid + j * CONS;
      if (idx < nfc) {
        const int e = idx / NF, q = idx - e * NF;
        const T uM = su[e * NP + sfm[q]];
        const T uP = g[idx];
        const double *gf = sgc + e * kCompactGeo64 + 9 + 4 * (q / (NF / 4));  // compact: the face's nx ny nz Fscale
        const T nsum = CP ? (T)(gf[0] + gf[1] + gf[2]) : sfc[idx] + sfc[FS + idx] + sfc[2 * FS + idx];
        const T fM = T(0.5) * uM * uM * nsum, fP = T(0.5) * uP * uP * nsum;
        const T an = fabs(nsum);
        const T lam = fmax(fabs(uM) * an, fabs(uP) * an);
        const T du = fM - (T(0.5) * (fM + fP) + T(0.5) * lam * (uM - uP));
        sf[e * NFS + q] = (CP ? (T)gf[3] : sfc[3 * FS + idx]) * du;
      }
    }
    if (!cons_sync_and<CONS>(ready)) {
      if (tid == 0) atomicExch(A.status, kStatusTimeoutCode);
      // the copies in flight land before the CTA goes: this tile's and the next tile's (the next tile's part B
      // was issued when every consumer had finished the previous tile, before this barrier)
      mbar_wait_bounded(&full[s], parity, kSpinLimit);
      mbar_wait_bounded(&fullb[s], parity, kSpinLimit);
      if (t + G < A.ntiles) {
        mbar_wait_bounded(&full[s ^ 1], ((k + 1) >> 1) & 1, kSpinLimit);
        mbar_wait_bounded(&fullb[s ^ 1], ((k + 1) >> 1) & 1, kSpinLimit);
      }
      return;
    }
    if (tid == 0) {
      mbar_arrive(&gfree[s]);  // the gathered traces of this tile are consumed
      // the metrics and face arrays of stage s are consumed too: tile t + 2G's part A streams in during (c)
      if (has2) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue_tile_a<N, CP, T>(A, t2, slot2, ring + s * C::STAGE_B, &full[s]);
      }
    }
    // (c) LIFT * flux on the tensor path, LSERK4 update in the epilogue
    {
      constexpr int CH = NW == 1 ? 3 : 2;  // accumulator chains per n-tile
      double c[NW][CH][2];
#pragma unroll
      for (int n = 0; n < NW; ++n)
#pragma unroll
        for (int h = 0; h < CH; ++h) c[n][h][0] = c[n][h][1] = 0.0;
#pragma unroll
      for (int kk = 0; kk < KL; ++kk)
#pragma unroll
        for (int n = 0; n < NW; ++n) {
          const double bv = be + 8 * n < ne ? sf[(be + 8 * n) * NFS + 4 * kk + acol] : 0.0;
          dmma(c[n][kk % CH][0], c[n][kk % CH][1], aL[kk], bv);
        }
#pragma unroll
      for (int n = 0; n < NW; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = ce + 8 * n + h;
          if (arow < NP && e < ne) {
            const int o = e * NP + arow;
            const int64_t gi = tl.node_base + o;
            const T rhs = vol[n][h] + (T)(c[n][0][h] + c[n][1][h] + (CH == 3 ? c[n][CH - 1][h] : 0.0));
            if (rhs_only) {
              __stcs(A.rhs_out + gi, rhs);
            } else {
              const T res = a * sr[o] + dt * rhs;
              __stcs(A.resu + gi, res);
              __stcs(A.u_out + gi, su[o] + b * res);
            }
          }
        }
    }
    // this warp has read the slot's u and resu (its loads returned: their values are in the stores above); the
    // last consumer warp to get here refills the slot's part B.  Slot s's counter is next touched by tile
    // t + 2G, which no warp reaches before every warp passed tile t + G's barrier, after this reset.
    __syncwarp();
    if (lane == 0) {
      __threadfence_block();
      if (atomicAdd(&done[s], 1) == CW - 1) {
        done[s] = 0;
        __threadfence_block();
        if (has2) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          issue_tile_b<N, CP, T>(A, t2, ring + s * C::STAGE_B, &fullb[s], rhs_only);
        }
      }
    }
    // rotate the descriptors at the end of the tile, where t2's load has long returned
    tcur = tnext;
    tnext = t2;
  }
}

template <int N, bool CP, typename T>
static void dmma_launch_n(const RhsArgs<T> &A, int rhs_only, int num_sms, cudaStream_t st, LaunchInfo *info) {
  using C = DmmaCfg<N, CP, T>;
  static_assert(C::SMEM <= 227 * 1024, "every order has the form");
  auto k = rhs_stage_dmma_kernel<N, CP, T>;
  const int per = resident_ctas(k, C::THREADS, C::SMEM, info);
  const int grid = std::min(A.ntiles, per * num_sms);
  if (info) *info = {grid, C::THREADS, (int)C::SMEM, per};
  if (grid > 0) launch_pdl(k, grid, C::THREADS, C::SMEM, st, A, rhs_only);
}

// Compact FP64 geometry of the compact form: per element slot the node-0 metrics and, per face, the first face
// point's nx, ny, nz and Fscale; an element whose values vary over its nodes or face points by more than 1e-6
// of the row's scale (the mixed stage's rule: node-to-node round-off of the FP64 metrics, where a curved
// element differs by O(h)) is counted in *bad (the form needs straight-sided elements).
__global__ void compact_geo64_kernel(CompactGeoArgs<double> g, double *out) {
  const int nfp = g.nf / 4;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < g.elem_total;
       x += (int64_t)gridDim.x * blockDim.x) {
    int p = 0;
    while (p + 1 < g.npart && g.elem_prefix[p + 1] <= x) ++p;
    const int64_t le = x - g.elem_prefix[p];
    const int64_t nb = g.node_off[p] + le * g.np, fb = g.face_off[p] + le * g.nf;
    double *o = out + (g.slot_prefix[p] + le) * kCompactGeo64;
    bool bad = false;
    for (int d = 0; d < 3; ++d) {
      double scale = 0.0;
      for (int q = 0; q < 3; ++q) scale = fmax(scale, fabs(g.geo[3 * d + q][nb]));
      for (int q = 0; q < 3; ++q) {
        const int m = 3 * d + q;
        const double v = g.geo[m][nb];
        for (int i = 1; i < g.np; ++i) bad |= !(fabs(g.geo[m][nb + i] - v) <= 1e-6 * scale);
        o[m] = v;
      }
    }
    for (int f = 0; f < 4; ++f) {
      const int64_t q0 = fb + f * nfp;
      const double ns = fmax(fabs(g.face[0][q0]), fmax(fabs(g.face[1][q0]), fabs(g.face[2][q0])));
      for (int c = 0; c < 4; ++c) {
        const double v = g.face[c][q0], sc = c < 3 ? ns : fabs(v);
        for (int q = 1; q < nfp; ++q) bad |= !(fabs(g.face[c][q0 + q] - v) <= 1e-6 * sc);
        o[9 + 4 * f + c] = v;
      }
    }
    if (bad) atomicAdd(g.bad, 1);
  }
}

void launch_compact_geo64(const CompactGeoArgs<double> &g, double *out, cudaStream_t st) {
  compact_geo64_kernel<<<592, 256, 0, st>>>(g, out);
  cuda_check(cudaGetLastError(), "compact_geo64_kernel launch");
}

template <bool CP, typename T>
static void dmma_launch(int N, const RhsArgs<T> &A, int rhs_only, int num_sms, cudaStream_t st, LaunchInfo *info) {
  switch (N) {
    case 1: dmma_launch_n<1, CP, T>(A, rhs_only, num_sms, st, info); break;
    case 2: dmma_launch_n<2, CP, T>(A, rhs_only, num_sms, st, info); break;
    case 3: dmma_launch_n<3, CP, T>(A, rhs_only, num_sms, st, info); break;
    case 4: dmma_launch_n<4, CP, T>(A, rhs_only, num_sms, st, info); break;
    case 5: dmma_launch_n<5, CP, T>(A, rhs_only, num_sms, st, info); break;
    default: throw Error(DGK_ERR_UNSUPPORTED, "stage on the FP64 tensor path: orders 1..5");
  }
}

template <typename T>
void launch_rhs_dmma(int N, const RhsArgs<T> &A, int rhs_only, int num_sms, cudaStream_t st, LaunchInfo *info) {
  if constexpr (std::is_same<T, double>::value)
    if (A.geoc) return dmma_launch<true, T>(N, A, rhs_only, num_sms, st, info);
  dmma_launch<false, T>(N, A, rhs_only, num_sms, st, info);
}

template <typename T>
int dmma_tile_elems(int N) {
  switch (N) {
    case 1: return DmmaShape<1, T>::TE;
    case 2: return DmmaShape<2, T>::TE;
    case 3: return DmmaShape<3, T>::TE;
    case 4: return DmmaShape<4, T>::TE;
    case 5: return DmmaShape<5, T>::TE;
    default: return 0;
  }
}

template void launch_rhs_dmma<double>(int, const RhsArgs<double> &, int, int, cudaStream_t, LaunchInfo *);
template void launch_rhs_dmma<float>(int, const RhsArgs<float> &, int, int, cudaStream_t, LaunchInfo *);
template int dmma_tile_elems<double>(int);
template int dmma_tile_elems<float>(int);

// ------------------------------------------------------------------------------------------------
// Volume derivative (`differentiate`) and the reference's volume-only computeRHS, orders 1..5.
//
// The stage's volume part alone: u and the nine metrics through a two-slot ring of bulk copies, Dr, Ds, Dt in registers
// (one warp per 8-row m-tile and NW n-tiles), products on the FP64 tensor path, results stored from the epilogue.  No
// data passes between warps, so a tile has one barrier, after which its slot is refilled.  Bound by HBM: two CTAs
// per SM with 45 KB slots at order 4.  Order 4, 32^3 x 6, FP64: 110-114 us (715 MB, 0.97 of the copy rate) from 176 with
// the register-staged form on the FP64 cores.  Tiles of 8 elements and three CTAs measured the same (117 against 119 us
// per call) with twice the tile list to build.
// ------------------------------------------------------------------------------------------------
template <int N, typename T>
struct DiffCfg {
  using O = Order<N>;
  static constexpr int NP = O::NP, TE = N == 1 ? 32 : 16, NW = N >= 3 ? 2 : 1;
  static constexpr int MT = (NP + 7) / 8, KT = (NP + 3) / 4;
  static constexpr int THREADS = 32 * MT * (TE / 8 / NW);
  static constexpr int AV = 16 / sizeof(T);
  static constexpr uint32_t NODE_B = TE * NP * sizeof(T) + 16, STAGE_B = 10 * NODE_B;
  static constexpr int NS = NODE_B / sizeof(T);
  static constexpr size_t SMEM = 2 * (size_t)STAGE_B + 16;
  static constexpr int PER = (int)(227 * 1024 / (SMEM + 1024));  // CTAs that share an SM by shared memory
  static constexpr int MINB = N == 5 || PER < 3 ? 2 : 3;
};

template <int N, typename T>
__device__ __forceinline__ void diff_issue(const DiffArgs<T> &A, const Tile &tl, char *stage, uint64_t *bar) {
  using C = DiffCfg<N, T>;
  const int ns = (int)(tl.node_base & (C::AV - 1));
  const uint32_t nb = round16((uint32_t)((tl.nelem * C::NP + ns) * sizeof(T)));
  mbar_expect_tx(bar, 10 * nb);
  bulk_g2s(stage, A.u + tl.node_base - ns, nb, bar);
#pragma unroll
  for (int m = 0; m < 9; ++m) bulk_g2s(stage + (1 + m) * C::NODE_B, A.geo[m] + tl.node_base - ns, nb, bar);
}

template <int N, typename T>
__global__ void __launch_bounds__(DiffCfg<N, T>::THREADS, DiffCfg<N, T>::MINB) diff_dmma_kernel(const DiffArgs<T> A) {
  using C = DiffCfg<N, T>;
  constexpr int NP = C::NP, KT = C::KT, MT = C::MT, NW = C::NW, NS = C::NS, LDD = pad_even(NP);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  char *ring = reinterpret_cast<char *>(smem_raw);
  uint64_t *full = reinterpret_cast<uint64_t *>(ring + 2 * C::STAGE_B);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, step = gridDim.x;
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const int mt = warp % MT, nt = warp / MT, acol = lane & 3;
  const int arow = mt * 8 + (lane >> 2);
  const int be = nt * NW * 8 + (lane >> 2), ce = nt * NW * 8 + 2 * acol;
  double aD[3][KT];
#pragma unroll
  for (int m = 0; m < 3; ++m)
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const int j = 4 * kk + acol;
      aD[m][kk] = (arow < NP && j < NP) ? A.D64[(m * NP + arow) * LDD + j] : 0.0;
    }
  pdl_wait();
  Tile t0 = A.tiles[blockIdx.x], t1{};
  if (blockIdx.x + step < A.ntiles) t1 = A.tiles[blockIdx.x + step];
  if (tid == 0) {
    diff_issue<N, T>(A, t0, ring, &full[0]);
    if (blockIdx.x + step < A.ntiles) diff_issue<N, T>(A, t1, ring + C::STAGE_B, &full[1]);
  }
  int k = 0;
  for (int t = blockIdx.x; t < A.ntiles; t += step, ++k) {
    const int s = k & 1;
    const bool has1 = t + step < A.ntiles, has2 = t + 2 * step < A.ntiles;
    if (tid == 0 && !has1) pdl_trigger();
    Tile t2{};
    if (has2) t2 = A.tiles[t + 2 * step];
    const bool ready = mbar_wait_bounded(&full[s], (uint32_t)(k >> 1) & 1u, kSpinLimit);
    const int ne = t0.nelem;
    const T *su = reinterpret_cast<const T *>(ring + s * C::STAGE_B) + (t0.node_base & (C::AV - 1));
    const T *sg = su + NS;
    double c[NW][3][2] = {};
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const int j = 4 * kk + acol;
#pragma unroll
      for (int n = 0; n < NW; ++n) {
        const double bv = (j < NP && be + 8 * n < ne) ? (double)su[(be + 8 * n) * NP + j] : 0.0;
#pragma unroll
        for (int m = 0; m < 3; ++m) dmma(c[n][m][0], c[n][m][1], aD[m][kk], bv);
      }
    }
#pragma unroll
    for (int n = 0; n < NW; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = ce + 8 * n + h;
        if (arow < NP && e < ne) {
          const int o = e * NP + arow;
          const int64_t gi = t0.node_base + o;
          const T ur = (T)c[n][0][h], us = (T)c[n][1][h], ut = (T)c[n][2][h];
          const T ux = sg[o] * ur + sg[3 * NS + o] * us + sg[6 * NS + o] * ut;
          const T uy = sg[NS + o] * ur + sg[4 * NS + o] * us + sg[7 * NS + o] * ut;
          const T uz = sg[2 * NS + o] * ur + sg[5 * NS + o] * us + sg[8 * NS + o] * ut;
          if (A.mode == 0) {
            __stcs(A.out[0] + gi, ux);
            __stcs(A.out[1] + gi, uy);
            __stcs(A.out[2] + gi, uz);
          } else {
            A.out[0][gi] = -su[o] * (ux + uy + uz);  // not streamed: an update reads it next
          }
        }
      }
    if (!__syncthreads_and(ready)) {  // the slot is free; a wait that gave up ends every thread here
      if (tid == 0) atomicExch(A.status, kStatusTimeoutCode);
      mbar_wait_bounded(&full[s], (uint32_t)(k >> 1) & 1u, kSpinLimit);  // copies in flight land before the CTA goes
      if (has1) mbar_wait_bounded(&full[s ^ 1], (uint32_t)((k + 1) >> 1) & 1u, kSpinLimit);
      return;
    }
    if (tid == 0 && has2) {
      fence_async_smem();
      diff_issue<N, T>(A, t2, ring + s * C::STAGE_B, &full[s]);
    }
    t0 = t1;
    t1 = t2;
  }
}

template <int N, typename T>
static void diff_launch_n(const DiffArgs<T> &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  using C = DiffCfg<N, T>;
  auto k = diff_dmma_kernel<N, T>;
  const int per = resident_ctas(k, C::THREADS, C::SMEM, info);
  const int grid = std::min(A.ntiles, per * num_sms);
  if (info) *info = {grid, C::THREADS, (int)C::SMEM, per};
  if (grid > 0) launch_pdl(k, grid, C::THREADS, C::SMEM, st, A);
}

template <typename T>
void launch_diff(int N, const DiffArgs<T> &A, int num_sms, cudaStream_t st, LaunchInfo *info) {
  switch (N) {
    case 1: diff_launch_n<1, T>(A, num_sms, st, info); break;
    case 2: diff_launch_n<2, T>(A, num_sms, st, info); break;
    case 3: diff_launch_n<3, T>(A, num_sms, st, info); break;
    case 4: diff_launch_n<4, T>(A, num_sms, st, info); break;
    case 5: diff_launch_n<5, T>(A, num_sms, st, info); break;
    default: throw Error(DGK_ERR_UNSUPPORTED, "order N must be 1..5");
  }
}
template void launch_diff<double>(int, const DiffArgs<double> &, int, cudaStream_t, LaunchInfo *);
template void launch_diff<float>(int, const DiffArgs<float> &, int, cudaStream_t, LaunchInfo *);

int diff_tile_elems(int N) { return N == 1 ? 32 : 16; }

}  // namespace dgk
