// Kernel bodies for tmc_kernels.cuh (included once per precision TU).
//
// Every kernel has two branches selected at compile time:
//  * T = double: the reference's arithmetic, element by element, in its
//    expression order (no FMA: the TU is compiled with -fmad=false);
//  * T = float: the fast path.  Neighbour indices and weights are loaded
//    first (fixed unrolled widths: maxEdges 6, maxEdges2 10, padded entries
//    carry zero weights or zero signs), then the neighbour gathers, then the
//    arithmetic, so each thread keeps tens of independent loads in flight.
//    GB300 executes FP64 at a small fraction of its FP32 rate, so the FP32
//    path keeps FP64 only for the gd tendency (from an FP32 two-sum
//    compensated flux divergence), the gd RK accumulation and the per-thread
//    invariant sums.
#pragma once

// Resident 256-thread blocks per SM the heavy ensemble kernels are built for
// (their register budget: 4 -> 64 registers, 3 -> 80).  On 512 level-6
// members, 4 for the flux, the cell pass without tracers and the final edge
// update takes the step from 9.85 to about 9.3 ms: the occupancy gain
// outweighs the few spilled bytes.
#ifndef TMC_FLUX_MIN_BLOCKS
#define TMC_FLUX_MIN_BLOCKS 4
#endif
#ifndef TMC_CELL_MIN_BLOCKS
#define TMC_CELL_MIN_BLOCKS 4
#endif
#ifndef TMC_FINAL_MIN_BLOCKS
#define TMC_FINAL_MIN_BLOCKS 4
#endif
// The same for the single-model cell pass (blocks of kCellBlock) and final
// edge update (blocks of up to kMaxBlock).  Level 9: the cell pass takes 139 us
// at 3 (80 registers) and 165 us at 4; the final pass 122 us at 2 (64
// registers, no spill), 129 us with no minimum (64 registers, 4 bytes
// spilled) and 176 us at 1 (120 registers).
#ifndef TMC_CELL_SINGLE_MIN_BLOCKS
#define TMC_CELL_SINGLE_MIN_BLOCKS 3
#endif
#ifndef TMC_FINAL_SINGLE_MIN_BLOCKS
#define TMC_FINAL_SINGLE_MIN_BLOCKS 2
#endif

#include <type_traits>

#include "tmc_fp64.cuh"
#include "tmc_kernels.cuh"

namespace tmc {

constexpr int kMaxBlock = 512;
constexpr int kMemberBlock = 256;  // block size limit of the ensemble (member-batched) kernels
constexpr int kCellBlock = 256;    // block size limit of the FP32 cell pass (register budget for 3 blocks/SM)
constexpr int kME = 6;    // unrolled maxEdges of the FP32 path
constexpr int kME2 = 10;  // unrolled maxEdges2 of the FP32 path

// Reduce N per-thread partial sums over the block and store region[r[k]][block]
// as (sum, 0).  FP32 sums: warps sum their lanes with a shuffle tree, warp 0
// sums the warp sums the same way.  FP64 sums: both levels in integers
// (f64::warp_sum), which leaves the FP64 pipe to the kernel's arithmetic: a
// shuffle tree costs five warp-wide FP64 instructions per warp and value, and
// warp 0 of every block sits on the same SM sub-partition, so an FP64 tail per
// block serialises behind the whole kernel.  The combination across blocks is
// k_finalize's.  Every thread of the block must call this (it synchronises).
template <class A>
__device__ __forceinline__ A lanes_sum(A w) {
  if constexpr (sizeof(A) == 8) {
    return f64::value(f64::warp_sum(w));
  } else {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) w += __shfl_down_sync(0xffffffffu, w, off);
    return w;
  }
}
template <class A, int N>
__device__ __forceinline__ void block_store(const A (&v)[N], const Partials& P, const int (&r)[N], int slot = -1) {
  if (slot < 0) slot = blockIdx.x;
  __shared__ A sm[N][kMaxBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const A w = lanes_sum(v[k]);
    if (lane == 0) sm[k][warp] = w;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const A w = lanes_sum((lane < nw) ? sm[k][lane] : A(0));
      if (lane == 0) {
        double* reg = P.region(r[k]);
        reg[2 * slot] = (double)w;
        reg[2 * slot + 1] = 0.0;
      }
    }
  }
  __syncthreads();
}

template <class T>
constexpr bool kF64 = std::is_same<T, double>::value;

// Programmatic dependent launch (Blk::pdl): the kernels of a small FP32 model's
// chain let the next one start at once (pdl_start) and wait for the previous one
// before they touch the state (pdl_wait), after the loads of the mesh where
// those come first.  In a launch without the attribute both do nothing.
template <class T, bool kB, int EPT>
constexpr bool kPdl = !kF64<T> && !kB && EPT == 1;
// the state of a dependent launch is another kernel's output until pdl_wait:
// plain loads, where a kernel alone reads its inputs through the read-only path
template <bool kDep, class T>
__device__ __forceinline__ T state_load(const T* p) {
  if constexpr (kDep)
    return *p;
  else
    return __ldg(p);
}

// The FP32 passes of one element per thread store the factors of the CRK4
// inner products and the vertex terms of the invariants, and no block sums:
// k_finalize_products sums them, and the other invariants from the state, in
// the order of the passes of kEPT elements per thread.
template <class T, int EPT>
constexpr bool kProducts = !kF64<T> && EPT == 1;

// metric in the arithmetic type: FP64 array in FP64 mode, FP32 copy otherwise
template <class T>
__device__ __forceinline__ const T* met_p(const double* d, const float* f) {
  if constexpr (kF64<T>)
    return d;
  else
    return f;
}
template <class T>
__device__ __forceinline__ T met(const double* d, const float* f, size_t i) {
  if constexpr (kF64<T>)
    return d[i];
  else
    return f[i];
}

// acc + a b of a global sum
__device__ __forceinline__ float fma_acc(float a, float b, float acc) { return acc + a * b; }
__device__ __forceinline__ double fma_acc(double a, double b, double acc) { return __fma_rn(a, b, acc); }
__device__ __forceinline__ float halve(float x) { return 0.5f * x; }
__device__ __forceinline__ double halve(double x) { return f64::half(x); }

template <class T>
__device__ __forceinline__ T sgn1(T x) {
  return copysign(T(1), x);
}

// FP32 error-free addition (TwoSum): hi + lo accumulates p exactly
__device__ __forceinline__ void two_sum_acc(float& hi, float& lo, float p) {
  const float t = __fadd_rn(hi, p);
  const float bp = __fsub_rn(t, hi);
  const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(t, bp)), __fsub_rn(p, bp));
  hi = t;
  lo = __fadd_rn(lo, err);
}

// block_store for compensated FP32 sums: the threads' (hi, lo) pairs are
// combined over each warp and then over the block with FP32 TwoSum
// arithmetic, and the block's pair is stored as (hi, lo) in FP64 (two
// conversions per block).  An FP64 shuffle tree costs ten FP64 instructions
// per warp, and GB300 runs each warp-wide FP64 instruction on a 2-lane pipe
// (16 cycles), which in the final edge update was most of the FP64 pipe's
// busy time.  Every thread of the block must call this (it synchronises).
template <int N>
__device__ __forceinline__ void block_store_ff(const float (&hi)[N], const float (&lo)[N], const Partials& P,
                                               const int (&r)[N], int slot = -1) {
  if (slot < 0) slot = blockIdx.x;
  __shared__ float sh[N][kMaxBlock / 32], sl[N][kMaxBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    float h = hi[k], l = lo[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const float oh = __shfl_down_sync(0xffffffffu, h, off), ol = __shfl_down_sync(0xffffffffu, l, off);
      two_sum_acc(h, l, oh);
      l = __fadd_rn(l, ol);
    }
    if (lane == 0) {
      sh[k][warp] = h;
      sl[k][warp] = l;
    }
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float h = (lane < nw) ? sh[k][lane] : 0.f, l = (lane < nw) ? sl[k][lane] : 0.f;
#pragma unroll
      for (int off = kMaxBlock / 64; off > 0; off >>= 1) {
        const float oh = __shfl_down_sync(0xffffffffu, h, off), ol = __shfl_down_sync(0xffffffffu, l, off);
        two_sum_acc(h, l, oh);
        l = __fadd_rn(l, ol);
      }
      if (lane == 0) {
        double* reg = P.region(r[k]);
        reg[2 * slot] = (double)h;
        reg[2 * slot + 1] = (double)l;
      }
    }
  }
  __syncthreads();
}

// block-strided loop: thread handles i = base + k*blockDim.x, k < EPT
#define TMC_FOR_AT(bx, EPT, i, n)                                                                         \
  for (int _k = 0, i = (bx) * (EPT * blockDim.x) + threadIdx.x; _k < EPT; ++_k, i += blockDim.x) \
    if (i < (n))
#define TMC_FOR_N(EPT, i, n) TMC_FOR_AT((int)blockIdx.x, EPT, i, n)
#define TMC_FOR_EPT(i, n) TMC_FOR_N(kEPT, i, n)

// x / 12
__device__ __forceinline__ float over12(float x) { return x / 12.f; }
__device__ __forceinline__ double over12(double x) { return f64::div_r(x, 12.0, 1.0 / 12.0); }

// Upwind correction of an edge value from two-sided polynomial-fit stencils
// (operators_mod.F90:423-472 for cells, :359-412 for vertices).  `f(i)`
// returns the field at stencil point i as T; ctr0/ctr1 are the two centres.
template <class T, class F>
__device__ __forceinline__ T upwind_edge(const DStencil& S2, const DStencil& S4, int order, T coef2, T coef4, int ne,
                                         int e, int ctr0, int ctr1, T fe, T sgn_of, T dist, F f) {
  if (order == 3 || order == 4) {
    T d0, d1;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const T fc = f(s == 0 ? ctr0 : ctr1);
      T acc = T(0);
      const int n = S2.count[(size_t)s * ne + e];
#pragma unroll 4
      for (int j = 0; j < n; ++j) {
        const size_t k = ((size_t)j * 2 + s) * ne + e;
        acc = acc + T(S2.w[k]) * (f(S2.idx[k]) - fc);
      }
      if (s == 0)
        d0 = acc;
      else
        d1 = acc;
    }
    fe = fe - over12(dist * dist * ((d0 + d1) - sgn1(sgn_of) * coef2 * (d1 - d0)));
  } else if (order == 5 || order == 6) {
    T a0, a1, b0, b1;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const T fc = f(s == 0 ? ctr0 : ctr1);
      T acc = T(0);
      int n = S2.count[(size_t)s * ne + e];
      for (int j = 0; j < n; ++j) {
        const size_t k = ((size_t)j * 2 + s) * ne + e;
        acc = acc + T(S2.w[k]) * (f(S2.idx[k]) - fc);
      }
      T acc4 = T(0);
      n = S4.count[(size_t)s * ne + e];
      for (int j = 0; j < n; ++j) {
        const size_t k = ((size_t)j * 2 + s) * ne + e;
        acc4 = acc4 + T(S4.w[k]) * (f(S4.idx[k]) - fc);
      }
      if (s == 0) {
        a0 = acc;
        b0 = acc4;
      } else {
        a1 = acc;
        b1 = acc4;
      }
    }
    fe = fe - dist * dist * (a0 + a1) / T(12) +
         (dist * dist) * (dist * dist) * ((b0 + b1) - sgn1(sgn_of) * coef4 * (b1 - b0)) / T(60);
  }
  return fe;
}

// sum_j deriv(j, side, e) (f(fit_j) - f(centre)) of one stencil side, in stencil order
template <class T, class F>
__device__ __forceinline__ T stencil_side(const DStencil& S, int ne, int e, int side, T fc, F f) {
  T acc = T(0);
  const int n = S.count[(size_t)side * ne + e];
  for (int j = 0; j < n; ++j) {
    const size_t k = ((size_t)j * 2 + side) * ne + e;
    acc = acc + T(S.w[k]) * (f(S.idx[k]) - fc);
  }
  return acc;
}

// ---------------------------------------------------------------------------
// edge_prep: gd_edge, u, mass flux F, tracer fluxes
// ---------------------------------------------------------------------------
// The cell-side values an edge preparation reads: gd (FP64, or the FP32
// shadow) and the tracer mass (FP64) or mixing-ratio shadow (FP32) of one
// state slot.
template <class T>
struct CellSrc {
  const double* gd;
  const float* gdf;
  const T* q;
  const float* qr;
  const double* ratio;  // FP64: mixing ratios [ntr][nc], or null (divide q by gd)
};

// The edge quantities of a stage that an edge preparation writes.
template <class T>
struct EdgeSet {
  T *gd_e, *u, *F, *Fq;
  double *sq, *hu, *ke, *ud;  // FP64 path
  float* uf;                  // FP64 path with upwind pv: u in FP32
};
template <class T>
__device__ __forceinline__ EdgeSet<T> edge_set(const StageIO<T>& S) {
  return {S.gd_e, S.u, S.F, S.Fq, S.sq, S.hu, S.ke, S.ud, S.uf};
}
template <class T>
__device__ __forceinline__ EdgeSet<T> next_edge_set(const StageIO<T>& S) {
  return {S.gd_e_nx, S.u_nx, S.F_nx, S.Fq_nx, S.sq_nx, S.hu_nx, S.ke_nx, S.ud_nx, S.uf_nx};
}

// Edge preparation of one edge (operators_mod.F90:93-104 c2e, :423-472 upwind
// correction with the sign of iap_u, :168-176 inverse IAP; the mass flux
// u*gd_edge of tmcore_swm_mod.F90:135; for tracers of order >= 3 the sg11
// edge value of adv_scheme_sg11_mod.F90:42-45 times the mass flux).
// g1, g2 are the two cells' gd in T, already loaded by the caller.
//
// FP64: the terms that the cell, vertex and flux passes sum are formed here,
// once per edge instead of once per use (two cells, two vertices, and the
// flux pass's square root and quotient over again): the signed sums of those
// passes take them with a sign flip, so the products' roundings are the
// reference's.  F holds u gd_edge dvEdge, Fq the tracers' terms, ke u^2
// areaEdge, ud u dcEdge, sq sqrt(gd_edge) and hu (u/2)/sqrt(gd_edge).  At
// about 64 cycles per warp-wide FP64 instruction the extra 64 bytes per edge
// are the cheaper side: a level-8 step with four tracers 5.29 -> 2.89 ms
// with the reciprocal quotients (tmc_fp64.cuh).
// ratios: C.ratio holds the tracers' mixing ratios of the two cells, else
// they are divided here (a state set from outside).
template <class T>
__device__ __forceinline__ void prep_edge(const DevMesh& M, const ModelOpt& O, int e, int c1, int c2, T ia, T g1,
                                          T g2, const CellSrc<T>& C, const EdgeSet<T>& X) {
  if constexpr (kF64<T>) {
    double ge = f64::half(g1 + g2);
    if (O.adv_order >= 3) {
      const double* gd = C.gd;
      ge = upwind_edge<T>(M.cell2, M.cell4, O.adv_order, T(O.cell_coef2), T(O.cell_coef4), M.ne, e, c1, c2, ge, ia,
                          M.dcEdge[e], [gd](int i) { return gd[i]; });
    }
    const double dv = M.dvEdge[e], dc = M.dcEdge[e], ae = M.areaEdge[e];
    const f64::SqrtR sq = f64::sqrt_r(ge);
    const double uu = f64::div_r(ia, sq.s, sq.r);
    const double Fv = uu * ge;
    X.gd_e[e] = ge;
    X.u[e] = uu;
    X.F[e] = Fv * dv;
    X.sq[e] = sq.s;
    X.hu[e] = f64::div_r(f64::half(uu), sq.s, sq.r);
    X.ke[e] = uu * uu * ae;
    X.ud[e] = uu * dc;
    if (X.uf) X.uf[e] = (float)uu;
    for (int k = 0; k < O.n_tracers; ++k) {
      double qe;
      if (C.ratio) {
        const double* r = C.ratio + (size_t)k * M.nc;
        qe = f64::half(r[c1] + r[c2]);
      } else {
        const double* q = C.q + (size_t)k * M.nc;
        qe = f64::half(q[c1] / g1 + q[c2] / g2);
      }
      if (O.tr_order >= 3) {
        const double* q = C.q + (size_t)k * M.nc;
        const double* gd = C.gd;
        qe = upwind_edge<T>(M.cell2, M.cell4, O.tr_order, T(O.tr_coef2), T(O.tr_coef4), M.ne, e, c1, c2, qe, ia, dc,
                            [q, gd](int i) { return q[i] / gd[i]; });
      }
      X.Fq[(size_t)k * M.ne + e] = Fv * qe * dv;
    }
  } else {
    T ge = T(0.5) * (g1 + g2);
    if (O.adv_order >= 3) {
      const float* gd = C.gdf;
      ge = upwind_edge<T>(M.cell2, M.cell4, O.adv_order, T(O.cell_coef2), T(O.cell_coef4), M.ne, e, c1, c2, ge, ia,
                          M.dcEdge_f[e], [gd](int i) { return gd[i]; });
    }
    const T sq = sqrt(ge);
    const T uu = ia / sq;
    const T Fv = uu * ge;
    if (X.gd_e) X.gd_e[e] = ge;
    X.u[e] = uu;
    X.F[e] = Fv;
    // second-order tracers are fluxed by k_cell directly (no per-edge flux stored)
    for (int k = 0; k < (O.tr_order >= 3 ? O.n_tracers : 0); ++k) {
      const float* qr = C.qr + (size_t)k * M.nc;
      T qe = 0.5f * (qr[c1] + qr[c2]);
      qe = upwind_edge<T>(M.cell2, M.cell4, O.tr_order, T(O.tr_coef2), T(O.tr_coef4), M.ne, e, c1, c2, qe, ia,
                          M.dcEdge_f[e], [qr](int i) { return qr[i]; });
      X.Fq[(size_t)k * M.ne + e] = Fv * qe;
    }
  }
}

template <class T>
__device__ __forceinline__ T energy_term(const DevMesh& M, int e, T ia) {
  if constexpr (kF64<T>)
    return ia * ia * M.areaEdge[e];  // tmcore_swm_mod.F90:229
  else
    return ia * ia * M.areaEdge_f[e];
}

// Stand-alone edge preparation of a state slot (the first stage after the
// state was set, the diagnostic pass, spatial_operators).
template <class T, bool kB, int EPT>
__global__ void __launch_bounds__(kMaxBlock) k_edge_prep(DevMesh M, ModelOpt O, StageIO<T> S0, Partials P0, int diag) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  double en = 0.0;
  const CellSrc<T> C{S.gd_in, S.gdf_in, S.q_in, S.qr_in, nullptr};
  TMC_FOR_N(EPT, e, M.ne) {
    const int c1 = M.cellsOnEdge[e], c2 = M.cellsOnEdge[M.ne + e];
    const T ia = S.iap_in[e];
    T g1, g2;
    if constexpr (kF64<T>) {
      g1 = S.gd_in[c1];
      g2 = S.gd_in[c2];
    } else {
      g1 = S.gdf_in[c1];
      g2 = S.gdf_in[c2];
    }
    prep_edge<T>(M, O, e, c1, c2, ia, g1, g2, C, edge_set(S));
    if (!kProducts<T, EPT> && diag) {
      if constexpr (kF64<T>)
        en = en + energy_term<T>(M, e, ia);
      else
        en += (double)energy_term<T>(M, e, ia);
    }
  }
  if (!kProducts<T, EPT> && diag) {
    const double v[1] = {en};
    const int r[1] = {R_EN_E};
    block_store<double, 1>(v, P, r);
  }
  if (kProducts<T, EPT> && diag && blockIdx.x == 0 && threadIdx.x == 0) *S.en64 = 1;
}

// ---------------------------------------------------------------------------
// cell: div of mass flux, kinetic energy, E, RK update of gd and tracers
// ---------------------------------------------------------------------------
// (kDep, here and below: a dependent launch)
template <class T, bool kB, int EPT, bool kDep>
__device__ __forceinline__ void cell_body(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S0, RKStage rk,
                                          const Partials& P0, int diag, int b0 = 0) {
  const int bx = (int)blockIdx.x - b0;  // this block among the cells' blocks
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  if constexpr (kDep) {
    pdl_start();
    pdl_wait();
  }
  T rip = T(0), r44 = T(0);
  double mass = 0.0, enc = 0.0;
  TMC_FOR_AT(bx, EPT, c, M.nc) {
    double t;  // gd tendency, FP64 in both modes
    double rA = 0.0;  // FP64: 1 / areaCell
    T tT, ke;
    int eidx[kME], cidx[kME];
    float nsg[kME];
    const int n = M.nEdgesOnCell[c];
    const int mode = rk.mode;
    // RK inputs before any store (see k_edge_flux)
    const double gold = (mode >= 1 && mode <= 3) ? S.gd_old[c] : 0.0;
    const double gacc = (mode >= 2) ? S.gd_acc[c] : 0.0;
    T tprev = T(0);
    if constexpr (kF64<T>)
      tprev = (mode >= 2) ? S.gd_tend[c] : 0.0;
    else
      tprev = (mode >= 2) ? S.tendf[c] : 0.f;
    const double gdin = diag ? S.gd_in[c] : 0.0, ghsd = diag ? S.ghs[c] : 0.0;
    if constexpr (kF64<T>) {
      // operators_mod.F90:40-55 (div_operator of u*gd_edge) and :206-221, in
      // order, from the edges' terms (prep_edge): one addition per edge and sum
      double s = 0.0, k = 0.0;
#pragma unroll 6
      for (int i = 0; i < n; ++i) {
        const int e = M.edgesOnCell[(size_t)i * M.nc + c];
        s = s + f64::with_sign(S.F[e], M.nSign[(size_t)i * M.nc + c]);
        k = k + S.ke[e];
      }
      const double A = M.areaCell[c];
      rA = M.invAreaCell[c];
      t = f64::div_r(-s, A, rA);
      tT = t;
      ke = f64::div_r(f64::half(f64::half(k)), A, rA);
      S.E[c] = ke + S.gd_in[c] + S.ghs[c];
      (void)eidx;
      (void)cidx;
      (void)nsg;
    } else {
      float uu[kME], Fv[kME], dv[kME], ae[kME];
      const bool tr_direct = O.n_tracers > 0 && O.tr_order == 2;
#pragma unroll
      for (int i = 0; i < kME; ++i) {
        eidx[i] = M.edgesOnCell[(size_t)i * M.nc + c];  // padded slots: index 0, sign 0
        nsg[i] = (float)M.nSign[(size_t)i * M.nc + c];
        cidx[i] = tr_direct ? M.cellsOnCell[(size_t)i * M.nc + c] : 0;
      }
#pragma unroll
      for (int i = 0; i < kME; ++i) {
        uu[i] = S.u[eidx[i]];
        Fv[i] = S.F[eidx[i]];
        dv[i] = M.dvEdge_f[eidx[i]];
        ae[i] = M.areaEdge_f[eidx[i]];
      }
      float hi = 0.f, lo = 0.f, k = 0.f;
#pragma unroll
      for (int i = 0; i < kME; ++i) {
        // the FP32 flux of an edge is bit-identical in its two cells; the two-sum
        // keeps their sum exact enough for mass conservation to FP64 round-off
        two_sum_acc(hi, lo, __fmul_rn(__fmul_rn(nsg[i], Fv[i]), dv[i]));
        k += fabsf(nsg[i]) * uu[i] * uu[i] * ae[i];
      }
      t = -((double)hi + (double)lo) * M.invAreaCell[c];
      tT = (float)t;
      ke = k * 0.25f * M.invAreaCell_f[c];
      S.E[c] = ke + S.gdf_in[c] + S.ghsf[c];
    }
    (void)n;
    const double Ad = M.areaCell[c];
    double gnext = 0.0;
    if constexpr (kF64<T>) {
      double* tb = S.gd_tend;
      switch (mode) {
        case 0:
          tb[c] = t;
          break;
        case 1:
          S.gd_acc[c] = t;
          tb[c] = t;
          gnext = gold + rk.a_dt * t;
          S.gd_next[c] = gnext;
          break;
        case 2:
        case 3: {
          rip = __fma_rn(tprev * t, Ad, rip);
          S.gd_acc[c] = __fma_rn(2.0, t, gacc);  // 2 t is exact
          tb[c] = t;
          gnext = gold + rk.a_dt * t;
          S.gd_next[c] = gnext;
          break;
        }
        case 4: {
          rip = __fma_rn(tprev * t, Ad, rip);
          const double tn = f64::div_r(gacc + t, 6.0, 1.0 / 6.0);
          S.gd_acc[c] = tn;
          r44 = __fma_rn(tn * tn, Ad, r44);
          tb[c] = t;
          break;
        }
      }
    } else {
      float* tb = S.tendf;
      const float Af = M.areaCell_f[c];
      switch (mode) {
        case 0:
          S.gd_tend[c] = t;
          tb[c] = tT;
          break;
        case 1:
          S.gd_acc[c] = t;
          tb[c] = tT;
          gnext = gold + rk.a_dt * t;
          S.gd_next[c] = gnext;
          S.gdf_next[c] = (float)gnext;
          break;
        case 2:
        case 3: {
          if constexpr (kProducts<T, EPT>)
            S.ipc[(size_t)(mode - 2) * M.nc + c] = tprev * tT;
          else
            rip += tprev * tT * Af;
          S.gd_acc[c] = gacc + 2.0 * t;
          tb[c] = tT;
          gnext = gold + rk.a_dt * t;
          S.gd_next[c] = gnext;
          S.gdf_next[c] = (float)gnext;
          break;
        }
        case 4: {
          const double tn = (gacc + t) * (1.0 / 6.0);
          S.gd_acc[c] = tn;
          const float tnf = (float)tn;
          if constexpr (kProducts<T, EPT>) {
            S.ipc[(size_t)2 * M.nc + c] = tprev * tT;
            S.ipc[(size_t)3 * M.nc + c] = tnf * tnf;
          } else {
            rip += tprev * tT * Af;
            r44 += tnf * tnf * Af;
          }
          tb[c] = tT;
          break;
        }
      }
    }
    // tracers, kTr at a time: loads and divergences first, then the stores
    constexpr int kTr = 4;
    double rg = 0.0;  // FP64: 1 / the next stage's gd
    if constexpr (kF64<T>)
      if (O.n_tracers > 0 && mode >= 1 && mode <= 3) rg = f64::recip(gnext);
    for (int q0 = 0; q0 < O.n_tracers; q0 += kTr) {
      T tq[kTr], qo[kTr], qa[kTr];
#pragma unroll
      for (int j = 0; j < kTr; ++j) {
        const int q = q0 + j;
        tq[j] = qo[j] = qa[j] = T(0);
        if (q >= O.n_tracers) continue;
        const size_t qi = (size_t)q * M.nc + c;
        qo[j] = (mode >= 1 && mode <= 3) ? S.q_old[qi] : T(0);
        qa[j] = (mode >= 2) ? S.q_acc[qi] : T(0);
        // Second-order tracers take the edge value from the two cells directly,
        // q_edge = (q(c1) + q(c2))/2, so no per-edge tracer flux is stored;
        // higher orders read the fluxes k_edge_prep wrote with the upwind
        // correction.  The FP64 path sums the edges' terms of prep_edge.
        if constexpr (kF64<T>) {
          double sq = 0.0;
#pragma unroll 6
          for (int i = 0; i < n; ++i) {
            const int e = M.edgesOnCell[(size_t)i * M.nc + c];
            sq = sq + f64::with_sign(S.Fq[(size_t)q * M.ne + e], M.nSign[(size_t)i * M.nc + c]);
          }
          tq[j] = f64::div_r(-sq, M.areaCell[c], rA);
        } else {
          float sq = 0.f;
          if (O.tr_order == 2) {
            const float qs = S.qr_in[qi];
#pragma unroll
            for (int i = 0; i < kME; ++i) {
              const float qn = S.qr_in[(size_t)q * M.nc + cidx[i]];
              sq += nsg[i] * S.F[eidx[i]] * (0.5f * (qs + qn)) * M.dvEdge_f[eidx[i]];
            }
          } else {
#pragma unroll
            for (int i = 0; i < kME; ++i)
              sq += nsg[i] * S.Fq[(size_t)q * M.ne + eidx[i]] * M.dvEdge_f[eidx[i]];
          }
          tq[j] = -sq * M.invAreaCell_f[c];
        }
      }
#pragma unroll
      for (int j = 0; j < kTr; ++j) {
        const int q = q0 + j;
        if (q >= O.n_tracers) continue;
        const size_t qi = (size_t)q * M.nc + c;
        T qnext = T(0);
        const T adt = T(rk.a_dt);
        switch (mode) {
          case 1:
            S.q_acc[qi] = tq[j];
            qnext = qo[j] + adt * tq[j];
            if constexpr (kF64<T>) S.q_next[qi] = qnext;  // FP32: the next stage reads the ratio only
            break;
          case 2:
          case 3:
            if constexpr (kF64<T>)
              S.q_acc[qi] = __fma_rn(2.0, tq[j], qa[j]);
            else
              S.q_acc[qi] = qa[j] + T(2) * tq[j];
            qnext = qo[j] + adt * tq[j];
            if constexpr (kF64<T>) S.q_next[qi] = qnext;
            break;
          case 4:
            if constexpr (kF64<T>)
              S.q_acc[qi] = f64::div_r(qa[j] + tq[j], 6.0, 1.0 / 6.0);
            else
              S.q_acc[qi] = (qa[j] + tq[j]) * (1.0f / 6.0f);
            break;
          default:
            S.q_acc[qi] = tq[j];
        }
        if (mode >= 1 && mode <= 3) {
          if constexpr (kF64<T>)
            S.ratio[qi] = f64::div_r(qnext, gnext, rg);
          else
            S.qr_next[qi] = qnext / (float)gnext;
        }
      }
    }
    if (!kProducts<T, EPT> && diag) {
      mass = __fma_rn(gdin, Ad, mass);
      enc = __fma_rn(gdin * __fma_rn(2.0, ghsd, gdin), Ad, enc);
    }
  }
  if (!kProducts<T, EPT> && rk.mode >= 2) {
    const T v[2] = {rip, r44};
    const int r[2] = {R_IP_C + 2 * (rk.mode - 2), R_44_C};
    block_store<T, 2>(v, P, r, bx);
  }
  if (!kProducts<T, EPT> && diag) {
    const double v[2] = {mass, enc};
    const int r[2] = {R_MASS, R_EN_C};
    block_store<double, 2>(v, P, r, bx);
  }
}
template <class T, bool kB, int EPT>
__global__ void __launch_bounds__(kMaxBlock) k_cell(DevMesh M, ModelOpt O, StageIO<T> S0, RKStage rk, Partials P0,
                                                    int diag) {
  cell_body<T, kB, EPT, false>(M, O, S0, rk, P0, diag);
}

// ---------------------------------------------------------------------------
// vertex: gd on vertices, vorticity, potential vorticity
// ---------------------------------------------------------------------------
template <class T, bool kB, int EPT, bool kDep>
__device__ __forceinline__ void vertex_body(const DevMesh& M, const StageIO<T>& S0, const Partials& P0, int diag) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  if constexpr (kDep) pdl_start();
  double pe = 0.0, av = 0.0;      // FP64 path
  float ph = 0.f, pl = 0.f, ah = 0.f, al = 0.f;  // FP32 path: compensated sums
  if constexpr (kF64<T>) {
    TMC_FOR_N(EPT, v, M.nv) {
      // operators_mod.F90:106-123 (c2v), :76-91 (curl), :262-270 (pv)
      double s = 0.0, gv = 0.0, kt[3];
      int ci[3], ei[3], ts[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ci[i] = M.cellsOnVertex[(size_t)i * M.nv + v];
        ei[i] = M.edgesOnVertex[(size_t)i * M.nv + v];
        ts[i] = M.tSign[(size_t)i * M.nv + v];
        kt[i] = M.kite[(size_t)i * M.nv + v];
      }
      const double At = M.areaTriangle[v], rAt = M.invAreaTriangle[v], fv = M.fVertex[v];
#pragma unroll
      for (int i = 0; i < 3; ++i) gv = gv + S.gd_in[ci[i]] * kt[i];
      gv = f64::div_r(gv, At, rAt);
#pragma unroll
      for (int i = 0; i < 3; ++i) s = s + f64::with_sign(S.ud[ei[i]], ts[i]);
      const double vo = f64::div_r(-s, At, rAt);
      const double ab = fv + vo;
      const double pv = f64::div_r(ab, gv, f64::recip(gv));
      S.pv_v[v] = pv;
      if (S.vor) S.vor[v] = vo;
      if (S.gd_v) S.gd_v[v] = gv;
      if (diag) {
        pe = __fma_rn(ab * pv, At, pe);  // gd_vertex pv^2 areaTriangle
        av = __fma_rn(ab, At, av);
      }
    }
  } else {
    // one vertex at a time: measured faster than batching the loads of the
    // thread's vertices (which costs occupancy for a pass with three gathers)
    // Every load is a read-only (non-coherent) load: nothing this kernel
    // stores aliases them, which lets the compiler issue a vertex's loads
    // ahead of the previous vertex's stores.
    TMC_FOR_N(EPT, v, M.nv) {
      int ci[3], ei[3];
      float kt[3], ts[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ci[i] = __ldg(M.cellsOnVertex + (size_t)i * M.nv + v);
        ei[i] = __ldg(M.edgesOnVertex + (size_t)i * M.nv + v);
        kt[i] = __ldg(M.kite_f + (size_t)i * M.nv + v);
        ts[i] = (float)__ldg(M.tSign + (size_t)i * M.nv + v);
      }
      // (with a dependent launch the state is another kernel's output until
      // pdl_wait, so its loads then are plain ones)
      float g[3], uu[3], dc[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) dc[i] = __ldg(M.dcEdge_f + ei[i]);
      const float iA = __ldg(M.invAreaTriangle_f + v);
      const float At = diag ? __ldg(M.areaTriangle_f + v) : 0.f;
      const float fv = __ldg(M.fVertex_f + v);
      if constexpr (kDep) pdl_wait();
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        g[i] = state_load<kDep>(S.gdf_in + ci[i]);
        uu[i] = state_load<kDep>(S.u + ei[i]);
      }
      const float gv = (g[0] * kt[0] + g[1] * kt[1] + g[2] * kt[2]) * iA;
      const float sv = ts[0] * uu[0] * dc[0] + ts[1] * uu[1] * dc[1] + ts[2] * uu[2] * dc[2];
      const float vo = -sv * iA;
      const float pv = (fv + vo) / gv;
      S.pv_v[v] = pv;
      if (S.vor) S.vor[v] = vo;
      if (S.gd_v) S.gd_v[v] = gv;
      if (diag) {
        // potential enstrophy and absolute vorticity (tmcore_swm_mod.F90:233-255)
        // from FP32 terms with compensated sums: FP64 terms made this launch
        // FP64-pipe bound
        if constexpr (kProducts<T, EPT>) {
          S.vterm[v] = gv * (pv * pv) * At;
          S.vterm[(size_t)M.nv + v] = vo * At;
        } else {
          two_sum_acc(ph, pl, gv * (pv * pv) * At);
          two_sum_acc(ah, al, vo * At);
          two_sum_acc(ah, al, fv * At);
        }
      }
    }
  }
  if (!kProducts<T, EPT> && diag) {
    const int r[2] = {R_PE, R_AV};
    if constexpr (kF64<T>) {
      const double vv[2] = {pe, av};
      block_store<double, 2>(vv, P, r);
    } else {
      const float h[2] = {ph, ah}, l[2] = {pl, al};
      block_store_ff<2>(h, l, P, r);
    }
  }
}
template <class T, bool kB, int EPT>
__global__ void __launch_bounds__(kMaxBlock) k_vertex(DevMesh M, StageIO<T> S0, Partials P0, int diag) {
  vertex_body<T, kB, EPT, false>(M, S0, P0, diag);
}

// pv on cells: scalar_v2c_interp_operator as a gather (operators_mod.F90:125-141)
template <class T>
__global__ void __launch_bounds__(kMaxBlock) k_v2c(DevMesh M, const T* pv_v0, T* pv_c0, long long msv, long long msc) {
  const T* pv_v = pv_v0 + blockIdx.y * msv;
  T* pv_c = pv_c0 + blockIdx.y * msc;
  TMC_FOR_EPT(c, M.nc) {
    const T A = T(M.areaCell[c]);
    T s = T(0);
    for (int k = M.v2c_start[c]; k < M.v2c_start[c + 1]; ++k) s = s + pv_v[M.v2c_vertex[k]] * T(M.v2c_kite[k]) / A;
    pv_c[c] = s;
  }
}

// ---------------------------------------------------------------------------
// edge_pv: PV on edges (calc_pv_on_edge, operators_mod.F90:273-412)
// ---------------------------------------------------------------------------
template <class T, bool kB, int EPT>
__global__ void __launch_bounds__(kMaxBlock) k_edge_pv(DevMesh M, ModelOpt O, StageIO<T> S0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const bool need_v = (O.pv_scheme >= 2) || (O.pv_scheme == 1 && O.apvm_weight != 0.0);
  if constexpr (kPdl<T, kB, EPT>) {
    pdl_start();
    if (need_v) pdl_wait();
  }
  if (!need_v) {
    // centred pv (APVM weight 0): all loads of the thread's EPT edges first
    const int e0 = blockIdx.x * (EPT * blockDim.x) + threadIdx.x;
    int v1[EPT], v2[EPT];
    T pe[EPT];
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int e = e0 + j * blockDim.x;
      v1[j] = e < M.ne ? M.verticesOnEdge[e] : 0;
      v2[j] = e < M.ne ? M.verticesOnEdge[M.ne + e] : 0;
    }
    if constexpr (kPdl<T, kB, EPT>) pdl_wait();
#pragma unroll
    for (int j = 0; j < EPT; ++j) pe[j] = halve(S.pv_v[v1[j]] + S.pv_v[v2[j]]);
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int e = e0 + j * blockDim.x;
      if (e < M.ne) S.pv_e[e] = pe[j];
    }
    return;
  }
  TMC_FOR_N(EPT, e, M.ne) {
    const int v1 = M.verticesOnEdge[e], v2 = M.verticesOnEdge[M.ne + e];
    const T p1 = S.pv_v[v1], p2 = S.pv_v[v2];
    T pe = halve(p1 + p2);
    T ve = T(0);
    if (need_v) {
      const int n = M.nEdgesOnEdge[e];
#pragma unroll 5
      for (int i = 0; i < n; ++i) {
        const size_t k = (size_t)i * M.ne + e;
        ve = ve + S.u[M.edgesOnEdge[k]] * met<T>(M.weightsOnEdge, M.weightsOnEdge_f, k);
      }
    }
    if (O.pv_scheme == 1) {
      if (O.apvm_weight != 0.0) {
        const int c1 = M.cellsOnEdge[e], c2 = M.cellsOnEdge[M.ne + e];
        const T a = ve * (p2 - p1) / met<T>(M.dvEdge, M.dvEdge_f, e);
        const T b = S.u[e] * (S.pv_c[c2] - S.pv_c[c1]) / met<T>(M.dcEdge, M.dcEdge_f, e);
        pe = pe - T(O.apvm_weight * O.dt) * (a + b);
      }
    } else if (O.pv_scheme == 2) {
      // correction direction of the conservative APVM (operators_mod.F90:336-341);
      // pv_edge stays the centred average until k_cons_apply
      const int c1 = M.cellsOnEdge[e], c2 = M.cellsOnEdge[M.ne + e];
      const T a = ve * (p2 - p1) / met<T>(M.dvEdge, M.dvEdge_f, e);
      const T b = S.u[e] * (S.pv_c[c2] - S.pv_c[c1]) / met<T>(M.dcEdge, M.dcEdge_f, e);
      S.dpv[e] = a + b;
    } else if (O.pv_scheme == 3) {
      const T* pv = S.pv_v;
      pe = upwind_edge<T>(M.vert2, M.vert4, O.interp_pv_order, T(O.vert_coef2), T(O.vert_coef4), M.ne, e, v1, v2,
                          pe, ve, met<T>(M.dvEdge, M.dvEdge_f, e), [pv](int i) { return pv[i]; });
    }
    S.pv_e[e] = pe;
  }
}

// Upwind pv on edges (pv_scheme 3, interp_pv_order 3 or 4;
// operators_mod.F90:359-412) in two passes.  The three edges of a vertex share
// the vertex's fit points and differ in their weights only, so k_vert_fit
// gathers the points once per vertex and sums the three second derivatives,
// each into its edge's side; k_edge_up adds the two sides.  Per edge that is 8
// gathers, 8 point indices and 12 differences in place of 24 each, on which
// the pass per edge was latency bound.  Us per step, pass per edge -> these:
// level 6 FP32 87 -> 72, FP64 305 -> 275; level 8 FP32 1115 -> 727 (the two
// passes 174 -> 88), FP64 3622 -> 3117.  Sums in stencil order.
// A point's index and its three weights are one 16-byte record in FP32 (as
// separate loads, 12 points at a time: 128 registers and 112 us for
// k_vert_fit alone at level 8).  Points in flight x resident blocks, level 8,
// both passes: 6 x 4 87.8 us, 4 x 6 87.3, 12 x 3 91.5; FP64 2 to 6 alike.
template <class T, bool kB, bool kDep>
__global__ void __launch_bounds__(256, kF64<T> ? 1 : 4) k_vert_fit(DevMesh M, StageIO<T> S0) {
  constexpr int kU = kF64<T> ? 4 : 6;  // points whose loads are in flight together
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const int v = blockIdx.x * blockDim.x + threadIdx.x, nv = M.nv;
  if constexpr (kDep) pdl_start();
  if (v >= nv) return;
  const int n = __ldg(M.vfit_n + v);
  if (kDep && n == 0) pdl_wait();
  T fc = T(0), acc[3] = {T(0), T(0), T(0)};
  if constexpr (!kDep) fc = __ldg(S.pv_v + v);
  for (int j0 = 0; j0 < n; j0 += kU) {
    int ix[kU];
    T w[3][kU], f[kU];
#pragma unroll
    for (int j = 0; j < kU; ++j) {
      const int q = min(j0 + j, n - 1);
      if constexpr (kF64<T>) {
        ix[j] = __ldg(M.vfit_idx + (size_t)q * nv + v);
#pragma unroll
        for (int k = 0; k < 3; ++k) w[k][j] = __ldg(M.vfit_w + ((size_t)q * 3 + k) * nv + v);
      } else {
        const float4 r = __ldg(M.vfit_rec + (size_t)q * nv + v);
        w[0][j] = r.x;
        w[1][j] = r.y;
        w[2][j] = r.z;
        ix[j] = __float_as_int(r.w);
      }
    }
    if constexpr (kDep) {  // after the first points' records
      if (j0 == 0) {
        pdl_wait();
        fc = S.pv_v[v];
      }
    }
#pragma unroll
    for (int j = 0; j < kU; ++j) f[j] = state_load<kDep>(S.pv_v + ix[j]);
#pragma unroll
    for (int j = 0; j < kU; ++j)
      if (j0 + j < n) {
        const T d = f[j] - fc;
#pragma unroll
        for (int k = 0; k < 3; ++k) acc[k] = acc[k] + w[k][j] * d;
      }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int e = __ldg(M.edgesOnVertex + (size_t)k * nv + v);
    const bool first = __ldg(M.tSign + (size_t)k * nv + v) > 0;  // v is the edge's first vertex
    S.dfit[(first ? (size_t)0 : (size_t)M.ne) + e] = acc[k];
  }
}

// The sign of the tangential velocity (:223-237) picks the upwind side.  FP64:
// it is decided by an FP32 sum wherever that exceeds the sum's error bound (n + 2
// roundings of 2^-24 of the magnitudes for n neighbours, of which a mesh has at
// most 64; the test asks for 128), else by the FP64 sum in the reference order:
// 20 FP64 instructions per edge less.
template <class T, bool kDep>
__device__ __forceinline__ T upwind_sign(const DevMesh& M, const StageIO<T>& S, int e) {
  const int ne = M.ne;
  if constexpr (kF64<T>) {
    const int n = M.nEdgesOnEdge[e];
    float s = 0.f, a = 0.f;
#pragma unroll 5
    for (int i = 0; i < n; ++i) {
      const float t = __fmul_rn(__ldg(S.uf + __ldg(M.edgesOnEdge + (size_t)i * ne + e)),
                                __ldg(M.weightsOnEdge_f + (size_t)i * ne + e));
      s = __fadd_rn(s, t);
      a = __fadd_rn(a, fabsf(t));
    }
    if (fabsf(s) > a * 0x1p-17f && a > 1e-25f && a < 1e30f) return s < 0.f ? -1.0 : 1.0;
    double ve = 0.0;
    for (int i = 0; i < n; ++i) {
      const size_t k = (size_t)i * ne + e;
      ve = ve + S.u[M.edgesOnEdge[k]] * M.weightsOnEdge[k];
    }
    return sgn1(ve);
  } else {
    int eo[kME2];
    float wo[kME2], uo[kME2], ve = 0.f;
#pragma unroll
    for (int i = 0; i < kME2; ++i) {
      eo[i] = __ldg(M.edgesOnEdge + (size_t)i * ne + e);  // padded slots: the edge itself, weight 0
      wo[i] = __ldg(M.weightsOnEdge_f + (size_t)i * ne + e);
    }
    if constexpr (kDep) pdl_wait();
#pragma unroll
    for (int i = 0; i < kME2; ++i) uo[i] = state_load<kDep>(S.u + eo[i]);
#pragma unroll
    for (int i = 0; i < kME2; ++i) ve = ve + uo[i] * wo[i];
    return sgn1(ve);
  }
}
template <class T, bool kB, bool kDep>
__global__ void __launch_bounds__(256) k_edge_up(DevMesh M, ModelOpt O, StageIO<T> S0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (kDep) pdl_start();
  if (e >= M.ne) return;
  const int v1 = __ldg(M.verticesOnEdge + e), v2 = __ldg(M.verticesOnEdge + M.ne + e);
  const T dist = __ldg(met_p<T>(M.dvEdge, M.dvEdge_f) + e);
  const T sg = upwind_sign<T, kDep>(M, S, e);  // (waits for the previous kernel)
  const T d0 = state_load<kDep>(S.dfit + e), d1 = state_load<kDep>(S.dfit + M.ne + e);
  const T p1 = state_load<kDep>(S.pv_v + v1), p2 = state_load<kDep>(S.pv_v + v2);
  S.pv_e[e] = halve(p1 + p2) - over12(dist * dist * ((d0 + d1) - sg * T(O.vert_coef2) * (d1 - d0)));
}

// ---------------------------------------------------------------------------
// conservative APVM (calc_pv_on_edge, pv_scheme 2, operators_mod.F90:318-357)
// ---------------------------------------------------------------------------
// calc_tangent_vor_flux (:239-260) of pv_edge and of the correction dpv; the
// factor w u gd_edge / 2 of a neighbour is shared by both sums
template <class T, bool kB>
__global__ void __launch_bounds__(kMaxBlock) k_cons_tvf(DevMesh M, StageIO<T> S0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  TMC_FOR_EPT(e, M.ne) {
    const int n = M.nEdgesOnEdge[e];
    const T pe = S.pv_e[e], dp = S.dpv[e];
    T a = T(0), b = T(0);
    for (int i = 0; i < n; ++i) {
      const size_t k = (size_t)i * M.ne + e;
      const int ep = M.edgesOnEdge[k];
      const T f = met<T>(M.weightsOnEdge, M.weightsOnEdge_f, k) * S.u[ep] * S.gd_e[ep] * T(0.5);
      a = a + f * (pe + S.pv_e[ep]);
      b = b + f * (dp + S.dpv[ep]);
    }
    S.pvf[e] = a;
    S.dpvf[e] = b;
  }
}

// per vertex: c2v of the gd tendency (:106-123), the curls of both tangent
// fluxes (calc_vor_tend_on_vertex :414-421), and the partial sums
// s1 = sum pv^2 tend_gd_v A, s2 = sum pv curl(pvf) A, s3 = sum pv curl(dpvf) A
template <class T, bool kB>
__global__ void __launch_bounds__(kMaxBlock) k_cons_vertex(DevMesh M, StageIO<T> S0, Partials P0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  double s1 = 0.0, s2 = 0.0, s3 = 0.0;
  TMC_FOR_EPT(v, M.nv) {
    if constexpr (kF64<T>) {
      const double At = M.areaTriangle[v];
      double g = 0.0, a = 0.0, b = 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i)
        g = g + S.gd_tend[M.cellsOnVertex[(size_t)i * M.nv + v]] * M.kite[(size_t)i * M.nv + v];
      g = g / At;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int e = M.edgesOnVertex[(size_t)i * M.nv + v];
        const double ts = (double)M.tSign[(size_t)i * M.nv + v];
        a = a + ts * S.pvf[e] * M.dcEdge[e];
        b = b + ts * S.dpvf[e] * M.dcEdge[e];
      }
      const double vt = (-a) / At, dvt = (-b) / At, pv = S.pv_v[v];
      s1 = s1 + pv * pv * g * At;
      s2 = s2 + pv * vt * At;
      s3 = s3 + pv * dvt * At;
    } else {
      const float iA = M.invAreaTriangle_f[v];
      float g = 0.f, a = 0.f, b = 0.f;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        g += S.tendf[M.cellsOnVertex[(size_t)i * M.nv + v]] * M.kite_f[(size_t)i * M.nv + v];
        const int e = M.edgesOnVertex[(size_t)i * M.nv + v];
        const float ts = (float)M.tSign[(size_t)i * M.nv + v];
        a += ts * S.pvf[e] * M.dcEdge_f[e];
        b += ts * S.dpvf[e] * M.dcEdge_f[e];
      }
      const double At = M.areaTriangle[v];
      const float pv = S.pv_v[v];
      s1 += (double)(pv * pv * (g * iA)) * At;
      s2 += (double)(pv * (-a * iA)) * At;
      s3 += (double)(pv * (-b * iA)) * At;
    }
  }
  const double vals[3] = {s1, s2, s3};
  const int r[3] = {R_C1, R_C2, R_C3};
  block_store<double, 3>(vals, P, r);
}

// pv_edge = pv_edge - eps dt dpv (:355)
template <class T, bool kB>
__global__ void __launch_bounds__(kMaxBlock) k_cons_apply(DevMesh M, ModelOpt O, StageIO<T> S0, const double* eps0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const double* eps = kB ? eps0 + (size_t)blockIdx.y * kDiagStride : eps0;
  const double ed = *eps * O.dt;
  TMC_FOR_EPT(e, M.ne) S.pv_e[e] = S.pv_e[e] - T(ed) * S.dpv[e];
}

// ---------------------------------------------------------------------------
// generic integrators: state update, combination of tendencies, inner products
// ---------------------------------------------------------------------------
// cells [0, nc) then edges [nc, nc + ne) in one index space
template <class T>
__global__ void __launch_bounds__(kMaxBlock) k_update(DevMesh M, int ntr, UpdateArgs<T> a) {
  const double coef = a.coef_dev ? *a.coef_dev : a.a_dt;
  const int n = M.nc + (a.tiap ? M.ne : 0);
  TMC_FOR_EPT(i, n) {
    if (i < M.nc) {
      const int c = i;
      const double g = a.gd_o[c] + coef * a.tgd[c];  // tmcore_swm_mod.F90:211
      a.gd_n[c] = g;
      if constexpr (!kF64<T>) a.gdf_n[c] = (float)g;
      for (int k = 0; k < ntr; ++k) {
        const size_t qi = (size_t)k * M.nc + c;
        const T q = a.q_o[qi] + T(coef) * a.tq[qi];
        a.q_n[qi] = q;
        if constexpr (!kF64<T>) a.qr_n[qi] = q / (float)g;
      }
    } else {
      const int e = i - M.nc;
      a.iap_n[e] = a.iap_o[e] + T(coef) * a.tiap[e];  // :210
    }
  }
}

template <class T>
__global__ void __launch_bounds__(kMaxBlock) k_combine(DevMesh M, int ntr, int scheme, CombineArgs<T> a,
                                                       Partials P) {
  // inner products of operators_mod.F90:187-194 per region, FP64 accumulation
  double ip[4] = {0.0, 0.0, 0.0, 0.0};
  const int ncb = grid_for(M.nc, blockDim.x);  // blocks [0, ncb) do cells, the rest edges
  const bool cells = (int)blockIdx.x < ncb;
  const int n = cells ? M.nc : M.ne;
  const int b0 = cells ? 0 : ncb;
  for (int j = 0; j < kEPT; ++j) {
    const int i = ((int)blockIdx.x - b0) * blockDim.x * kEPT + j * blockDim.x + threadIdx.x;
    if (i >= n) break;
    double t[4], w;
    if (cells) {
      for (int k = 0; k < 4; ++k) t[k] = a.tgd[k] ? a.tgd[k][i] : 0.0;
      w = M.areaCell[i];
    } else {
      for (int k = 0; k < 4; ++k) t[k] = a.tiap[k] ? (double)a.tiap[k][i] : 0.0;
      w = M.areaEdge[i];
    }
    if (scheme == 3) {  // PC2: <t0,t1>, <t1,t1>
      ip[0] = ip[0] + t[0] * t[1] * w;
      ip[3] = ip[3] + t[1] * t[1] * w;
      continue;
    }
    double tn;
    if (scheme == 1) {  // CRK3 (time_scheme_mod.F90:90-100)
      tn = (t[0] + 4.0 * t[1] + t[2]) / 6.0;
      ip[0] = ip[0] + t[0] * t[1] * w;
      ip[1] = ip[1] + t[0] * t[2] * w;
      ip[2] = ip[2] + t[1] * t[2] * w;
    } else {  // CRK4 (:140-150)
      tn = (t[0] + 2.0 * t[1] + 2.0 * t[2] + t[3]) / 6.0;
      ip[0] = ip[0] + t[0] * t[1] * w;
      ip[1] = ip[1] + t[1] * t[2] * w;
      ip[2] = ip[2] + t[2] * t[3] * w;
    }
    if (cells) {
      a.tgd[0][i] = tn;
      for (int q = 0; q < ntr; ++q) {
        const size_t qi = (size_t)q * M.nc + i;
        const T q0 = a.tq[0][qi], q1 = a.tq[1][qi], q2 = a.tq[2][qi];
        if (scheme == 1) {
          a.tq[0][qi] = (q0 + T(4) * q1 + q2) / T(6);
        } else {
          const T q3 = a.tq[3][qi];
          a.tq[0][qi] = (q0 + T(2) * q1 + T(2) * q2 + q3) / T(6);
        }
      }
    } else if (a.tiap[0]) {
      if constexpr (kF64<T>) {
        a.tiap[0][i] = tn;
      } else {
        tn = (double)(T)tn;
        a.tiap[0][i] = (T)tn;
      }
    }
    if (cells || a.tiap[0]) ip[3] = ip[3] + tn * tn * w;
  }
  const int base = cells ? R_IP_C : R_IP_E;
  const int r4 = cells ? R_44_C : R_44_E;
  const int r[4] = {base, base + 2, base + 4, r4};
  // partial slot: the block index within its half, cells [0, ncb), edges [0, neb)
  block_store<double, 4>(ip, P, r, (int)blockIdx.x - b0);
}

// Launch KERNEL<T, kB, EPT> over n elements of every member: the
// member-batched variant (kB = true, FP32 only) when the stage has several
// ensemble members, else the single-member code, which addresses its arrays
// straight from the kernel parameters, with b.ept elements per thread.
#define TMC_LAUNCH(KERNEL, n, ...)                                                              \
  do {                                                                                          \
    if constexpr (!kF64<T>) {                                                                   \
      if (S.members > 1) {                                                                      \
        KERNEL<T, true, kEPT><<<dim3(grid_for(n, b.bs), nmem(S)), b.bs, 0, st>>>(__VA_ARGS__); \
        break;                                                                                  \
      }                                                                                         \
    }                                                                                           \
    if (b.ept == 1)                                                                             \
      launch(KERNEL<T, false, 1>, grid_for(n, b), b, st, __VA_ARGS__);                          \
    else                                                                                        \
      KERNEL<T, false, kEPT><<<grid_for(n, b), b.bs, 0, st>>>(__VA_ARGS__);                     \
  } while (0)
// the same for kernels of kEPT elements per thread only
#define TMC_LAUNCH_4(KERNEL, n, ...)                                                       \
  do {                                                                                     \
    if constexpr (!kF64<T>) {                                                              \
      if (S.members > 1) {                                                                 \
        KERNEL<T, true><<<dim3(grid_for(n, bs), nmem(S)), bs, 0, st>>>(__VA_ARGS__);      \
        break;                                                                             \
      }                                                                                    \
    }                                                                                      \
    KERNEL<T, false><<<grid_for(n, bs), bs, 0, st>>>(__VA_ARGS__);                         \
  } while (0)

template <class T>
void launch_cons_apvm(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, Partials P, double* diag_out, int bs,
                      cudaStream_t st) {
  TMC_LAUNCH_4(k_cons_tvf, M.ne, M, S);
  TMC_LAUNCH_4(k_cons_vertex, M.nv, M, S, P);
  launch_cons_eps(P, grid_for(M.nv, bs), O.dt, diag_out, st, (int)nmem(S));
  TMC_LAUNCH_4(k_cons_apply, M.ne, M, O, S, diag_out + 10);
}

template <class T>
void launch_update(const DevMesh& M, int ntr, const UpdateArgs<T>& a, int bs, cudaStream_t st) {
  const int n = M.nc + (a.tiap ? M.ne : 0);
  k_update<T><<<grid_for(n, bs), bs, 0, st>>>(M, ntr, a);
}

template <class T>
void launch_combine(const DevMesh& M, int ntr, int scheme, const CombineArgs<T>& a, Partials P, int bs,
                    cudaStream_t st) {
  const int g = grid_for(M.nc, bs) + grid_for(M.ne, bs);
  k_combine<T><<<g, bs, 0, st>>>(M, ntr, scheme, a, P);
}

// ---------------------------------------------------------------------------
// edge_flux: q.F_perp, gradient of E, iap_u tendency, RK update, inner products
// ---------------------------------------------------------------------------
// kMode: the stage of a second-order model (adv_order 2, no
// flux_4th_order_correct) as a constant, or kGeneral for the others with the
// stage at run time.  As a constant it takes the branches out from between a
// thread's loads; FP32 also averages gd_edge again instead of loading it (the
// edge preparation does not store it), and the tendencies of stages 1 and 4
// are not stored: stage 1's is the accumulator, stage 4's is not read.  Level
// 9, four tracers, us per pass: flux 201.7 -> 189.9, cell 134.7 -> 124.5
// (cell_fast_body), final 107.7 -> 98.5.
constexpr int kGeneral = -1;
template <class T, bool kB, int EPT, int kMode>
__device__ __forceinline__ void edge_flux_body(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S0, RKStage rk,
                                               const Partials& P0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  if constexpr (kPdl<T, kB, EPT>) pdl_start();
  T rip = T(0), r44 = T(0);  // FP32 path: FP32 products and per-thread sums, FP64 across warps
  constexpr bool kPlain = kMode != kGeneral;
  const int mode = kPlain ? kMode : rk.mode;
  TMC_FOR_N(EPT, e, M.ne) {
    // Loads that depend on no other load come first, before any store: a load
    // issued after a store through a pointer the compiler must assume aliases
    // would wait a full memory round trip.
    const int c1 = M.cellsOnEdge[e], c2 = M.cellsOnEdge[M.ne + e];
    const T ae = (mode >= 2) ? met<T>(M.areaEdge, M.areaEdge_f, e) : T(0);
    int ep[kME2];
    float w[kME2];
    T dc;
    if constexpr (!kF64<T>) {
#pragma unroll
      for (int i = 0; i < kME2; ++i) {
        const size_t k = (size_t)i * M.ne + e;
        ep[i] = M.edgesOnEdge[k];  // padded entries: own edge with weight 0
        w[i] = M.weightsOnEdge_f[k];
      }
      dc = M.dcEdge_f[e];
    } else {
      dc = M.dcEdge[e];
    }
    if constexpr (kPdl<T, kB, EPT>) pdl_wait();
    const T pe = S.pv_e[e];
    T uu = T(0), ge = T(0), sq = T(0), hu = T(0);
    if constexpr (kF64<T>) {
      sq = S.sq[e];
      hu = S.hu[e];
      if (!kPlain && O.adv_order >= 3) uu = S.u[e];
    } else {
      uu = S.u[e];
      if constexpr (kPlain)
        ge = 0.5f * (S.gdf_in[c1] + S.gdf_in[c2]);
      else
        ge = S.gd_e[e];
    }
    const T tp0 = (mode >= (kPlain ? 3 : 2)) ? S.iap_tend[e] : T(0);
    const T accv = (mode >= 2) ? S.iap_acc[e] : T(0);
    const T oldv = (mode >= 1 && mode <= 3) ? S.iap_old[e] : T(0);
    const T tp = (kPlain && mode == 2) ? accv : tp0;
    // the next stage's gd on the two cells (written by this stage's k_cell)
    const bool fuse = kPlain ? (mode >= 1 && mode <= 3) : (S.u_nx != nullptr);
    T gn1 = T(0), gn2 = T(0);
    if (fuse) {
      if constexpr (kF64<T>) {
        gn1 = S.gd_next[c1];
        gn2 = S.gd_next[c2];
      } else {
        gn1 = S.gdf_next[c1];
        gn2 = S.gdf_next[c2];
      }
    }
    T s = T(0), tge, dEdx;
    if constexpr (kF64<T>) {
      // calc_tangent_vor_flux (operators_mod.F90:239-260), in order
      // (its factor 1/2 taken out of the sum: powers of two round alike)
      const int n = M.nEdgesOnEdge[e];
#pragma unroll 5
      for (int i = 0; i < n; ++i) {
        const size_t k = (size_t)i * M.ne + e;
        const int ep = M.edgesOnEdge[k];
        s = s + M.weightsOnEdge[k] * S.u[ep] * S.gd_e[ep] * (pe + S.pv_e[ep]);
      }
      s = f64::half(s);
      dEdx = f64::div_r(S.E[c2] - S.E[c1], dc, M.invDcEdge[e]);
      tge = f64::half(S.gd_tend[c1] + S.gd_tend[c2]);
    } else {
      const float E1 = S.E[c1], E2 = S.E[c2], t1 = S.tendf[c1], t2 = S.tendf[c2];
      float Fv[kME2], pp[kME2];
#pragma unroll
      for (int i = 0; i < kME2; ++i) {
        Fv[i] = S.F[ep[i]];
        pp[i] = S.pv_e[ep[i]];
      }
#pragma unroll
      for (int i = 0; i < kME2; ++i) s += w[i] * Fv[i] * (0.5f * (pe + pp[i]));
      dEdx = (E2 - E1) / dc;
      tge = 0.5f * (t1 + t2);
    }
    if (!kPlain && O.flux4) {
      // flux_4th_order_correct (tmcore_swm_mod.F90:183-195): third derivatives
      // of E on the two cells' fit3 stencils
      const T* Ev = S.E;
      auto fE = [Ev](int i) { return Ev[i]; };
      const T d1 = stencil_side<T>(M.cell3, M.ne, e, 0, Ev[c1], fE);
      const T d2 = stencil_side<T>(M.cell3, M.ne, e, 1, Ev[c2], fE);
      dEdx = dEdx - (d2 - d1) * dc / T(24);
    }
    const T ut = s - dEdx;
    if (!kPlain && O.adv_order >= 3) {
      // the upwind side is the sign of the stage's iap_u (tmcore_swm_mod.F90:107-108);
      // u = iap_u / sqrt(gd_edge) carries the same sign bit, and unlike iap_u it
      // is always stored (the fused stages keep the next iap_u in registers)
      if constexpr (kF64<T>) {
        const double* gt = S.gd_tend;
        tge = upwind_edge<T>(M.cell2, M.cell4, O.adv_order, T(O.cell_coef2), T(O.cell_coef4), M.ne, e, c1, c2, tge,
                             uu, dc, [gt](int i) { return gt[i]; });
      } else {
        const float* gt = S.tendf;
        tge = upwind_edge<T>(M.cell2, M.cell4, O.adv_order, T(O.cell_coef2), T(O.cell_coef4), M.ne, e, c1, c2, tge,
                             uu, dc, [gt](int i) { return gt[i]; });
      }
    }
    // calc_u_tend_on_edge (tmcore_swm_mod.F90:155-201)
    T it;
    if constexpr (kF64<T>) {
      it = sq * ut + hu * tge;  // sqrt(gd_edge) and (u/2) / sqrt(gd_edge) of prep_edge
    } else {
      sq = sqrt(ge);
      it = sq * ut + T(0.5) * uu / sq * tge;
    }
    T* tb = S.iap_tend;
    T inext = T(0);  // iap_u of the next stage (update_state, tmcore_swm_mod.F90:210)
    switch (mode) {
      case 0:
        tb[e] = it;
        break;
      case 1:
        S.iap_acc[e] = it;
        if (!kPlain) tb[e] = it;
        inext = oldv + T(rk.a_dt) * it;
        break;
      case 2:
      case 3: {
        if constexpr (kProducts<T, EPT>)
          S.ipe[(size_t)(mode - 2) * M.ne + e] = tp * it;
        else
          rip = fma_acc(tp * it, ae, rip);
        if constexpr (kF64<T>)
          S.iap_acc[e] = __fma_rn(2.0, it, accv);  // 2 t is exact
        else
          S.iap_acc[e] = accv + T(2) * it;
        tb[e] = it;
        inext = oldv + T(rk.a_dt) * it;
        break;
      }
      case 4: {
        if constexpr (kProducts<T, EPT>)
          S.ipe[(size_t)(mode - 2) * M.ne + e] = tp * it;
        else
          rip = fma_acc(tp * it, ae, rip);
        T tn;
        if constexpr (kF64<T>)
          tn = f64::div_r(accv + it, 6.0, 1.0 / 6.0);
        else
          tn = (accv + it) * (1.0f / 6.0f);
        S.iap_acc[e] = tn;
        if constexpr (kProducts<T, EPT>)
          S.ipe[(size_t)3 * M.ne + e] = tn * tn;
        else
          r44 = fma_acc(tn * tn, ae, r44);
        if (!kPlain) tb[e] = it;
        break;
      }
    }
    if (fuse) {
      // edge preparation of the next stage from its gd and iap_u
      const CellSrc<T> C{S.gd_next, S.gdf_next, S.q_next, S.qr_next, S.ratio};
      prep_edge<T>(M, O, e, c1, c2, inext, gn1, gn2, C, next_edge_set(S));
    } else if (mode >= 1 && mode <= 3) {
      S.iap_next[e] = inext;
    }
  }
  if constexpr (kProducts<T, EPT>) return;
  if (mode >= 2) {
    const T v[2] = {rip, r44};
    const int r[2] = {R_IP_E + 2 * (mode - 2), R_44_E};
    block_store<T, 2>(v, P, r);
  }
}

// the single-model kernel, and the ensemble kernel (member = blockIdx.y) with
// its register budget capped so that member pointers do not halve occupancy
// (two blocks of 512, 64 registers: left to itself the compiler takes 40 for
// the FP32 stages, which holds their loads back, and up to 104 for the FP64
// stages, which leaves the FP64 pipe too few warps: level 8 402 -> 419 us)
template <class T, int EPT, int kMode>
__global__ void __launch_bounds__(kMaxBlock, 2) k_edge_flux(DevMesh M, ModelOpt O, StageIO<T> S0, RKStage rk, Partials P0) {
  edge_flux_body<T, false, EPT, kMode>(M, O, S0, rk, P0);
}
template <class T, int kMode>
__global__ void __launch_bounds__(kMemberBlock, TMC_FLUX_MIN_BLOCKS) k_edge_flux_members(DevMesh M, ModelOpt O, StageIO<T> S0, RKStage rk,
                                                                    Partials P0) {
  edge_flux_body<T, true, kEPT, kMode>(M, O, S0, rk, P0);
}
// f with the stage as a constant, or kGeneral
template <class F>
inline void on_mode(bool plain, int mode, F&& f) {
  switch (plain ? mode : kGeneral) {
    case 0: f(std::integral_constant<int, 0>()); break;
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    default: f(std::integral_constant<int, kGeneral>());
  }
}

// new = old + (beta dt) t_new (update_state, tmcore_swm_mod.F90:203-213)
// Cells: gd and tracer mass of state(old) in place, and their FP32 shadows.
template <class T, bool kB, int EPT>
__global__ void __launch_bounds__(kMaxBlock) k_final_cells(DevMesh M, ModelOpt O, StageIO<T> S0, const double* diag0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const double* diag = kB ? diag0 + (size_t)blockIdx.y * kDiagStride : diag0;
  if constexpr (kPdl<T, kB, EPT>) {
    pdl_start();
    pdl_wait();
  }
  const double bdt = diag[9];
  // all loads of the thread's EPT cells before any store (a load after a
  // store through a possibly aliasing pointer waits a full round trip)
  const int i0 = blockIdx.x * (EPT * blockDim.x) + threadIdx.x;
  double* gd = const_cast<double*>(S.gd_old);
  double g[EPT];
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    const int i = i0 + j * blockDim.x;
    g[j] = i < M.nc ? gd[i] + bdt * S.gd_acc[i] : 0.0;
  }
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    const int i = i0 + j * blockDim.x;
    if (i >= M.nc) continue;
    gd[i] = g[j];
    if constexpr (!kF64<T>) const_cast<float*>(S.gdf_in)[i] = (float)g[j];
  }
  T* qq = const_cast<T*>(S.q_old);
  double rg[EPT];  // FP64: 1 / gd
  for (int q = 0; q < O.n_tracers; ++q) {
    T qn[EPT];
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int i = i0 + j * blockDim.x;
      const size_t qi = (size_t)q * M.nc + i;
      qn[j] = i < M.nc ? qq[qi] + T(bdt) * S.q_acc[qi] : T(0);
    }
    if constexpr (kF64<T>)
      if (q == 0)
#pragma unroll
        for (int j = 0; j < EPT; ++j) rg[j] = f64::recip(g[j]);
#pragma unroll
    for (int j = 0; j < EPT; ++j) {
      const int i = i0 + j * blockDim.x;
      if (i >= M.nc) continue;
      const size_t qi = (size_t)q * M.nc + i;
      qq[qi] = qn[j];
      if constexpr (kF64<T>)
        S.ratio[qi] = f64::div_r(qn[j], g[j], rg[j]);
      else
        const_cast<float*>(S.qr_in)[qi] = qn[j] / (float)g[j];
    }
  }
}

// Edges: iap_u of state(old) in place, then the edge preparation of the next
// step's first stage (into S.gd_e/u/F/Fq) and the edge part of the total
// energy of the new state (tmcore_swm_mod.F90:229) for the next step's
// invariants.
template <class T, bool kB, int EPT>
__global__ void __launch_bounds__(kB ? kMemberBlock : kMaxBlock, kB ? TMC_FINAL_MIN_BLOCKS : TMC_FINAL_SINGLE_MIN_BLOCKS)
    k_final_edges(DevMesh M, ModelOpt O, StageIO<T> S0, const double* diag0, Partials P0) {
  const StageIO<T> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  const double* diag = kB ? diag0 + (size_t)blockIdx.y * kDiagStride : diag0;
  if constexpr (kPdl<T, kB, EPT>) {
    pdl_start();
    pdl_wait();
  }
  const double bdt = diag[9];
  double en = 0.0;
  const CellSrc<T> C{S.gd_old, S.gdf_in, S.q_old, S.qr_in, S.ratio};
  // loads of all EPT edges first (see k_final_cells)
  const int e0 = blockIdx.x * (EPT * blockDim.x) + threadIdx.x;
  T* iap = const_cast<T*>(S.iap_old);
  int c1[EPT], c2[EPT];
  T ia[EPT], g1[EPT], g2[EPT], ae[EPT];
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    const int e = e0 + j * blockDim.x;
    const bool in = e < M.ne;
    c1[j] = in ? M.cellsOnEdge[e] : 0;
    c2[j] = in ? M.cellsOnEdge[M.ne + e] : 0;
    ia[j] = in ? iap[e] + T(bdt) * S.iap_acc[e] : T(0);
    ae[j] = in ? met<T>(M.areaEdge, M.areaEdge_f, e) : T(0);  // for the energy, loaded before any store
  }
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    if constexpr (kF64<T>) {
      g1[j] = S.gd_old[c1[j]];
      g2[j] = S.gd_old[c2[j]];
    } else {
      g1[j] = S.gdf_in[c1[j]];
      g2[j] = S.gdf_in[c2[j]];
    }
  }
  float eh = 0.f, el = 0.f;  // FP32 path: the thread's few terms, compensated
#pragma unroll
  for (int j = 0; j < EPT; ++j) {
    const int e = e0 + j * blockDim.x;
    if (e >= M.ne) continue;
    iap[e] = ia[j];
    prep_edge<T>(M, O, e, c1[j], c2[j], ia[j], g1[j], g2[j], C, edge_set(S));
    // energy_term (tmcore_swm_mod.F90:229) with areaEdge already loaded
    if constexpr (kF64<T>)
      en = __fma_rn(ia[j] * ia[j], ae[j], en);
    else
      two_sum_acc(eh, el, ia[j] * ia[j] * ae[j]);
  }
  if constexpr (kProducts<T, EPT>) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *S.en64 = 0;
    return;
  }
  const int r[1] = {R_EN_E};
  if constexpr (kF64<T>) {
    const double v[1] = {en};
    block_store<double, 1>(v, P, r);
  } else {
    const float h[1] = {eh}, l[1] = {el};
    block_store_ff<1>(h, l, P, r);
  }
}

template <class T>
__global__ void k_gather(int n, const double* src, const int32_t* n2o, T* dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = T(src[n2o[i]]);
}
template <class T>
__global__ void k_scatter(int n, const T* src, const int32_t* n2o, double* dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[n2o[i]] = (double)src[i];
}
template <class T>
__global__ void k_iap_from_u(int ne, const double* gd_e, const double* u, T* iap) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ne) iap[i] = T(sqrt(gd_e[i]) * u[i]);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
inline int nblk(int n, int bs) { return (n + bs - 1) / bs; }


template <class T>
void launch_edge_prep(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, Partials P, bool diag, Blk b,
                      cudaStream_t st) {
  TMC_LAUNCH(k_edge_prep, M.ne, M, O, S, P, diag ? 1 : 0);
}
// The second-order tracer terms of the FP32 cell pass (the mass-weighted
// form d(gd q)/dt = div_operator(F q_edge), q_edge the mean of the two
// cells' mixing ratios): the tendency of each tracer of one cell ...
template <int NTR, int NQ>
__device__ __forceinline__ void tracer_tend_f(const float (&ns)[kME], const float (&Fv)[kME], const float (&dv)[kME],
                                              const float (&qs)[NQ], const float (&qn)[NQ][kME], float invAf,
                                              float (&tq)[NQ]) {
#pragma unroll
  for (int j = 0; j < NTR; ++j) {
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < kME; ++i) sq += ns[i] * Fv[i] * (0.5f * (qs[j] + qn[j][i])) * dv[i];
    tq[j] = __fmul_rn(-sq, invAf);  // a tendency, not a term of an FMA
  }
}
// ... and its RK update (mode as RKStage; gnf the stage's next gd in FP32).
// The next stage reads the mixing ratio only (and q_old, q_acc), so the
// stage's tracer mass itself is not stored.
template <int NTR, int NQ>
__device__ __forceinline__ void tracer_update_f(const StageIO<float>& S, size_t nc, int c, int mode, float adt,
                                                const float (&tq)[NQ], const float (&qo)[NQ], const float (&qa)[NQ],
                                                float gnf) {
#pragma unroll
  for (int j = 0; j < NTR; ++j) {
    const size_t qi = (size_t)j * nc + c;
    if (mode == 1) {
      S.q_acc[qi] = tq[j];
    } else if (mode <= 3) {
      S.q_acc[qi] = qa[j] + 2.f * tq[j];
    } else {
      S.q_acc[qi] = (qa[j] + tq[j]) * (1.0f / 6.0f);
    }
    if (mode <= 3) {
      const float qnext = qo[j] + adt * tq[j];
      S.qr_next[qi] = qnext / gnf;
    }
  }
}

// FP32 cell pass of the CRK4 stages (modes 1-4) with NTR second-order
// tracers: every load is issued before the first store, in two waves
// (indices and the cell's own values, then the gathers of the edges' u, F,
// dvEdge, areaEdge and of the neighbours' tracer mixing ratios), so one cell
// costs two memory round trips.  Same arithmetic as the FP32 branch of k_cell.
// kMode as in edge_flux_body; with tracers the constant stages form the mass
// flux from u and the two cells' gd (whose index the tracers need anyway)
// instead of gathering it.
template <int NTR, bool kB, int EPT, int kMode, bool kDep>
__device__ __forceinline__ void cell_fast_body(const DevMesh& M, const StageIO<float>& S0, RKStage rk,
                                               const Partials& P0, int diag, int b0 = 0) {
  const int bx = (int)blockIdx.x - b0;  // this block among the cells' blocks
  if constexpr (kDep) pdl_start();
  const StageIO<float> S = kB ? S0.at(blockIdx.y) : S0;
  const Partials P = kB ? P0.at(blockIdx.y) : P0;
  constexpr int NQ = NTR > 0 ? NTR : 1;
  float rip = 0.f, r44 = 0.f;
  double mass = 0.0;
  float eh = 0.f, el = 0.f;
  constexpr bool kPlain = kMode != kGeneral;
  const int mode = kPlain ? kMode : rk.mode;
  TMC_FOR_AT(bx, EPT, c, M.nc) {
    int ei[kME], ci[kME];
    float ns[kME];
#pragma unroll
    for (int i = 0; i < kME; ++i) {
      ei[i] = M.edgesOnCell[(size_t)i * M.nc + c];
      ns[i] = (float)M.nSign[(size_t)i * M.nc + c];
      ci[i] = NTR > 0 ? M.cellsOnCell[(size_t)i * M.nc + c] : 0;
    }
    const double invA = M.invAreaCell[c];
    const float invAf = M.invAreaCell_f[c];
    const float Af = (mode >= 2) ? M.areaCell_f[c] : 0.f;
    float uu[kME], Fv[kME], dv[kME], ae[kME], qn[NQ][kME];
    if constexpr (kDep) {  // the mesh's values, then the previous kernel's
#pragma unroll
      for (int i = 0; i < kME; ++i) {
        dv[i] = M.dvEdge_f[ei[i]];
        ae[i] = M.areaEdge_f[ei[i]];
      }
      pdl_wait();
    }
    const double gold = (mode <= 3) ? S.gd_old[c] : 0.0;
    const double gacc = (mode >= 2) ? S.gd_acc[c] : 0.0;
    const float tprev = (kPlain && mode == 2) ? (float)gacc : (mode >= 2) ? S.tendf[c] : 0.f;
    const float gdf = S.gdf_in[c], ghf = S.ghsf[c];
    float qs[NQ], qo[NQ], qa[NQ];
#pragma unroll
    for (int j = 0; j < NTR; ++j) {
      const size_t qi = (size_t)j * M.nc + c;
      qs[j] = S.qr_in[qi];
      qo[j] = (mode <= 3) ? S.q_old[qi] : 0.f;
      qa[j] = (mode >= 2) ? S.q_acc[qi] : 0.f;
    }
    double gdin = 0.0, Ad = 0.0;
    float Afd = 0.f;
    if (diag) {
      gdin = S.gd_in[c];
      Ad = M.areaCell[c];
      Afd = M.areaCell_f[c];
    }
#pragma unroll
    for (int i = 0; i < kME; ++i) {
      uu[i] = S.u[ei[i]];
      Fv[i] = kPlain && NTR > 0 ? S.gdf_in[ci[i]] : S.F[ei[i]];
      if constexpr (!kDep) {
        dv[i] = M.dvEdge_f[ei[i]];
        ae[i] = M.areaEdge_f[ei[i]];
      }
    }
#pragma unroll
    for (int j = 0; j < NTR; ++j)
#pragma unroll
      for (int i = 0; i < kME; ++i) qn[j][i] = S.qr_in[(size_t)j * M.nc + ci[i]];
    if constexpr (kPlain && NTR > 0)  // u gd_edge, the operations of prep_edge
#pragma unroll
      for (int i = 0; i < kME; ++i) Fv[i] = __fmul_rn(uu[i], __fmul_rn(0.5f, __fadd_rn(gdf, Fv[i])));
    // divergence of the mass flux (two-sum), kinetic energy, E
    float hi = 0.f, lo = 0.f, k = 0.f;
#pragma unroll
    for (int i = 0; i < kME; ++i) {
      two_sum_acc(hi, lo, __fmul_rn(__fmul_rn(ns[i], Fv[i]), dv[i]));
      k += fabsf(ns[i]) * uu[i] * uu[i] * ae[i];
    }
    const double t = __dmul_rn(-((double)hi + (double)lo), invA);
    const float tT = (float)t;
    S.E[c] = k * 0.25f * invAf + gdf + ghf;
    float tq[NQ];
    tracer_tend_f<NTR, NQ>(ns, Fv, dv, qs, qn, invAf, tq);
    double gnext = 0.0;
    switch (mode) {
      case 1:
        S.gd_acc[c] = t;
        S.tendf[c] = tT;
        gnext = gold + rk.a_dt * t;
        break;
      case 2:
      case 3:
        if constexpr (kProducts<float, EPT>)
          S.ipc[(size_t)(mode - 2) * M.nc + c] = tprev * tT;
        else
          rip += tprev * tT * Af;
        S.gd_acc[c] = gacc + 2.0 * t;
        S.tendf[c] = tT;
        gnext = gold + rk.a_dt * t;
        break;
      default: {
        const double tn = (gacc + t) * (1.0 / 6.0);
        S.gd_acc[c] = tn;
        const float tnf = (float)tn;
        if constexpr (kProducts<float, EPT>) {
          S.ipc[(size_t)2 * M.nc + c] = tprev * tT;
          S.ipc[(size_t)3 * M.nc + c] = tnf * tnf;
        } else {
          rip += tprev * tT * Af;
          r44 += tnf * tnf * Af;
        }
        S.tendf[c] = tT;
      }
    }
    const float gnf = (float)gnext;
    if (mode <= 3) {
      S.gd_next[c] = gnext;
      S.gdf_next[c] = gnf;
    }
    tracer_update_f<NTR, NQ>(S, M.nc, c, mode, (float)rk.a_dt, tq, qo, qa, gnf);
    if (!kProducts<float, EPT> && diag) {
      // total mass from the FP64 gd; the cell part of the total energy
      // (gd^2 + 2 gd ghs) areaCell (tmcore_swm_mod.F90:215-231) from FP32
      // terms with a compensated sum (an FP64 term would cost four FP64
      // operations per cell at 1/64 of the FP32 rate)
      mass = mass + gdin * Ad;
      two_sum_acc(eh, el, gdf * (gdf + 2.f * ghf) * Afd);
    }
  }
  if (!kProducts<float, EPT> && mode >= 2) {
    const float v[2] = {rip, r44};
    const int r[2] = {R_IP_C + 2 * (mode - 2), R_44_C};
    block_store<float, 2>(v, P, r);
  }
  if (!kProducts<float, EPT> && diag) {
    const double v[2] = {mass, (double)eh + (double)el};
    const int r[2] = {R_MASS, R_EN_C};
    block_store<double, 2>(v, P, r);
  }
}

template <int NTR, int EPT, int kMode>
__global__ void __launch_bounds__(kCellBlock, TMC_CELL_SINGLE_MIN_BLOCKS) k_cell_fast(DevMesh M, StageIO<float> S0, RKStage rk, Partials P0,
                                                         int diag) {
  cell_fast_body<NTR, false, EPT, kMode, false>(M, S0, rk, P0, diag);
}
// The tracer terms of the FP32 cell pass alone, for a stage whose cell pass
// ran tracer-free (k_cell_fast<0>): the same loads and the same arithmetic
// (tracer_tend_f, tracer_update_f) as k_cell_fast<NTR>, with the stage's next
// gd in FP32 read back from S.gdf_next.  Single member.
template <int NTR, int EPT>
__global__ void __launch_bounds__(kCellBlock) k_tracers_fast(DevMesh M, StageIO<float> S, RKStage rk) {
  const int mode = rk.mode;
  TMC_FOR_N(EPT, c, M.nc) {
    int ei[kME], ci[kME];
    float ns[kME];
#pragma unroll
    for (int i = 0; i < kME; ++i) {
      ei[i] = M.edgesOnCell[(size_t)i * M.nc + c];
      ns[i] = (float)M.nSign[(size_t)i * M.nc + c];
      ci[i] = M.cellsOnCell[(size_t)i * M.nc + c];
    }
    const float invAf = M.invAreaCell_f[c];
    const float gnf = (mode <= 3) ? S.gdf_next[c] : 0.f;
    float qs[NTR], qo[NTR], qa[NTR];
#pragma unroll
    for (int j = 0; j < NTR; ++j) {
      const size_t qi = (size_t)j * M.nc + c;
      qs[j] = S.qr_in[qi];
      qo[j] = (mode <= 3) ? S.q_old[qi] : 0.f;
      qa[j] = (mode >= 2) ? S.q_acc[qi] : 0.f;
    }
    float Fv[kME], dv[kME], qn[NTR][kME];
#pragma unroll
    for (int i = 0; i < kME; ++i) {
      Fv[i] = S.F[ei[i]];
      dv[i] = M.dvEdge_f[ei[i]];
    }
#pragma unroll
    for (int j = 0; j < NTR; ++j)
#pragma unroll
      for (int i = 0; i < kME; ++i) qn[j][i] = S.qr_in[(size_t)j * M.nc + ci[i]];
    float tq[NTR];
    tracer_tend_f<NTR, NTR>(ns, Fv, dv, qs, qn, invAf, tq);
    tracer_update_f<NTR, NTR>(S, M.nc, c, mode, (float)rk.a_dt, tq, qo, qa, gnf);
  }
}

template <int NTR, int kMode>
__global__ void __launch_bounds__(kMemberBlock, NTR == 0 ? TMC_CELL_MIN_BLOCKS : 3) k_cell_fast_members(DevMesh M, StageIO<float> S0, RKStage rk,
                                                                    Partials P0, int diag) {
  cell_fast_body<NTR, true, kEPT, kMode, false>(M, S0, rk, P0, diag);
}

template <class T>
void launch_cell(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, RKStage rk, Partials P, bool diag, Blk b,
                 cudaStream_t st) {
  if constexpr (!kF64<T>) {
    const bool fast = rk.mode >= 1 && rk.mode <= 4 && launch_cell_is_fast(O);
    const int dg = diag ? 1 : 0;
    auto run = [&](auto ntr) {
      constexpr int N = decltype(ntr)::value;
      on_mode(!S.gd_e, rk.mode, [&](auto m) {
        constexpr int kMode = decltype(m)::value;
        if constexpr (kMode != 0) {
          if (S.members > 1)
            k_cell_fast_members<N, kMode><<<dim3(grid_for(M.nc, b.bs), nmem(S)), b.bs, 0, st>>>(M, S, rk, P, dg);
          else if (b.ept == 1)
            k_cell_fast<N, 1, kMode><<<grid_for(M.nc, b), b.bs, 0, st>>>(M, S, rk, P, dg);
          else
            k_cell_fast<N, kEPT, kMode><<<grid_for(M.nc, b), b.bs, 0, st>>>(M, S, rk, P, dg);
        }
      });
    };
    if (fast) {
      switch (O.n_tracers) {
        case 0: run(std::integral_constant<int, 0>()); return;
        case 1: run(std::integral_constant<int, 1>()); return;
        case 2: run(std::integral_constant<int, 2>()); return;
        case 4: run(std::integral_constant<int, 4>()); return;
        default: break;
      }
    }
  }
  TMC_LAUNCH(k_cell, M.nc, M, O, S, rk, P, diag ? 1 : 0);
}
template <class T>
void launch_tracers_fast(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, RKStage rk, Blk b,
                         cudaStream_t st) {
  if constexpr (!kF64<T>) {
    auto run = [&](auto ntr) {
      constexpr int N = decltype(ntr)::value;
      if (b.ept == 1)
        k_tracers_fast<N, 1><<<grid_for(M.nc, b), b.bs, 0, st>>>(M, S, rk);
      else
        k_tracers_fast<N, kEPT><<<grid_for(M.nc, b), b.bs, 0, st>>>(M, S, rk);
    };
    switch (O.n_tracers) {
      case 1: run(std::integral_constant<int, 1>()); return;
      case 2: run(std::integral_constant<int, 2>()); return;
      case 4: run(std::integral_constant<int, 4>()); return;
      default: return;
    }
  }
}
template <class T>
void launch_vertex(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, Partials P, bool diag, Blk b,
                   cudaStream_t st) {
  TMC_LAUNCH(k_vertex, M.nv, M, S, P, diag ? 1 : 0);
}
template <class T>
void launch_edge_pv(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, Blk b, cudaStream_t st) {
  if ((O.pv_scheme == 1 && O.apvm_weight != 0.0) || O.pv_scheme == 2 || O.need_pv_c)
    k_v2c<T><<<dim3(grid_for(M.nc, b.bs), nmem(S)), b.bs, 0, st>>>(M, S.pv_v, S.pv_c, S.msv, S.msc);
  if (M.vfit_n) {
    const int bs = b.bs < 256 ? b.bs : 256;
    const dim3 gv(nblk(M.nv, bs), nmem(S)), ge(nblk(M.ne, bs), nmem(S));
    if constexpr (!kF64<T>) {
      if (S.members > 1) {
        k_vert_fit<T, true, false><<<gv, bs, 0, st>>>(M, S);
        k_edge_up<T, true, false><<<ge, bs, 0, st>>>(M, O, S);
        return;
      }
    }
    if constexpr (!kF64<T>) {
      if (b.pdl) {
        launch(k_vert_fit<T, false, true>, gv.x, Blk(bs, 1, true), st, M, S);
        launch(k_edge_up<T, false, true>, ge.x, Blk(bs, 1, true), st, M, O, S);
        return;
      }
    }
    k_vert_fit<T, false, false><<<gv, bs, 0, st>>>(M, S);
    k_edge_up<T, false, false><<<ge, bs, 0, st>>>(M, O, S);
    return;
  }
  TMC_LAUNCH(k_edge_pv, M.ne, M, O, S);
}
template <class T>
void launch_edge_flux(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, RKStage rk, Partials P, Blk b,
                      cudaStream_t st) {
  // FP32 models that are not second order, and the conservative APVM, store gd_edge
  const bool plain = kF64<T> ? O.adv_order == 2 && !O.flux4 : !S.gd_e;
  on_mode(plain, rk.mode, [&](auto m) {
    constexpr int kMode = decltype(m)::value;
    if constexpr (!kF64<T>) {
      if (S.members > 1) {
        k_edge_flux_members<T, kMode><<<dim3(grid_for(M.ne, b.bs), nmem(S)), b.bs, 0, st>>>(M, O, S, rk, P);
        return;
      }
    }
    if (b.ept == 1)
      launch(k_edge_flux<T, 1, kMode>, grid_for(M.ne, b), b, st, M, O, S, rk, P);
    else
      k_edge_flux<T, kEPT, kMode><<<grid_for(M.ne, b), b.bs, 0, st>>>(M, O, S, rk, P);
  });
}
template <class T>
void launch_final_update(const DevMesh& M, const ModelOpt& O, const StageIO<T>& S, const double* diag, Partials P,
                         Blk b, cudaStream_t st) {
  TMC_LAUNCH(k_final_cells, M.nc, M, O, S, diag);
  TMC_LAUNCH(k_final_edges, M.ne, M, O, S, diag, P);
}
template <class T>
void launch_gather(int n, const double* src, const int32_t* n2o, T* dst, cudaStream_t st) {
  k_gather<T><<<nblk(n, 256), 256, 0, st>>>(n, src, n2o, dst);
}
template <class T>
void launch_scatter(int n, const T* src, const int32_t* n2o, double* dst, cudaStream_t st) {
  k_scatter<T><<<nblk(n, 256), 256, 0, st>>>(n, src, n2o, dst);
}
template <class T>
void launch_iap_from_u(int ne, const double* gd_e, const double* u, T* iap, cudaStream_t st) {
  k_iap_from_u<T><<<nblk(ne, 256), 256, 0, st>>>(ne, gd_e, u, iap);
}

// mpas_reconstruct_1d (mpas_vector_reconstruction.F90:207-261), reference order
template <class T>
__global__ void k_reconstruct(DevMesh M, const T* u, double* uX, double* uY, double* uZ, double* zon, double* mer) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= M.nc) return;
  double x = 0.0, y = 0.0, z = 0.0;
  for (int i = 0; i < M.nEdgesOnCell[c]; ++i) {
    const double ue = (double)u[M.edgesOnCell[(size_t)i * M.nc + c]];
    x = x + M.recon[((size_t)0 * M.me + i) * M.nc + c] * ue;
    y = y + M.recon[((size_t)1 * M.me + i) * M.nc + c] * ue;
    z = z + M.recon[((size_t)2 * M.me + i) * M.nc + c] * ue;
  }
  if (uX) uX[c] = x;
  if (uY) uY[c] = y;
  if (uZ) uZ[c] = z;
  const double clat = M.cell_trig[c], slat = M.cell_trig[(size_t)M.nc + c];
  const double clon = M.cell_trig[(size_t)2 * M.nc + c], slon = M.cell_trig[(size_t)3 * M.nc + c];
  if (zon) zon[c] = -x * slon + y * clon;
  if (mer) mer[c] = -(x * clon + y * slon) * slat + z * clat;
}

template <class T>
__global__ void k_to_f64(size_t n, const T* src, double* dst) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (double)src[i];
}

template <class T>
void launch_reconstruct(const DevMesh& M, const T* u, double* uX, double* uY, double* uZ, double* zonal,
                        double* meridional, cudaStream_t st) {
  k_reconstruct<T><<<nblk(M.nc, 256), 256, 0, st>>>(M, u, uX, uY, uZ, zonal, meridional);
}
template <class T>
void launch_to_f64(size_t n, const T* src, double* dst, cudaStream_t st) {
  k_to_f64<T><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, src, dst);
}

// the cell passes (their many stage and tracer variants compile beside the rest)
#define TMC_INSTANTIATE_CELL(T) \
  template void launch_cell<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, RKStage, Partials, bool, Blk, \
                               cudaStream_t);                                                                     \
  template void launch_tracers_fast<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, RKStage, Blk,           \
                                       cudaStream_t);

#define TMC_INSTANTIATE(T)                                                                                        \
  template void launch_gather<T>(int, const double*, const int32_t*, T*, cudaStream_t);                          \
  template void launch_scatter<T>(int, const T*, const int32_t*, double*, cudaStream_t);                         \
  template void launch_iap_from_u<T>(int, const double*, const double*, T*, cudaStream_t);                       \
  template void launch_edge_prep<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, Partials, bool, Blk,     \
                                    cudaStream_t);                                                                \
  template void launch_vertex<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, Partials, bool, Blk,        \
                                 cudaStream_t);                                                                   \
  template void launch_edge_pv<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, Blk, cudaStream_t);        \
  template void launch_edge_flux<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, RKStage, Partials, Blk,  \
                                    cudaStream_t);                                                                \
  template void launch_final_update<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, const double*,         \
                                       Partials, Blk, cudaStream_t);                                             \
  template void launch_cons_apvm<T>(const DevMesh&, const ModelOpt&, const StageIO<T>&, Partials, double*, int,   \
                                    cudaStream_t);                                                                \
  template void launch_update<T>(const DevMesh&, int, const UpdateArgs<T>&, int, cudaStream_t);                 \
  template void launch_reconstruct<T>(const DevMesh&, const T*, double*, double*, double*, double*, double*,   \
                                      cudaStream_t);                                                            \
  template void launch_to_f64<T>(size_t, const T*, double*, cudaStream_t);                                       \
  template void launch_combine<T>(const DevMesh&, int, int, const CombineArgs<T>&, Partials, int, cudaStream_t);

}  // namespace tmc
