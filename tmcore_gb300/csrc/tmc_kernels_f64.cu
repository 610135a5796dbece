// FP64 instantiation (compiled with -fmad=false: no FMA contraction, so each
// element follows the reference's IEEE operation order), the reduction
// finaliser, the FP32 shadow helpers and the single-operator kernels used for
// parity.
#include <algorithm>

#include "tmc_kernels_impl.cuh"

namespace tmc {

TMC_INSTANTIATE(double)
TMC_INSTANTIATE_CELL(double)

struct FinalizeArgs {
  int counts[R_COUNT];
  double totalArea, sumAreaTriangle, dt;
  int step, diag, conserve, scheme;
  int split;  // blocks per region (1..kFinSplit)
};

// The sum of `count` per-block partials (hi, lo pairs) by one block, as a
// (hi, lo) pair in the lanes of warp 0: per-thread FP64 sums of a few
// partials, then integer sums of the threads (f64::warp_sum).
__device__ f64::HiLo region_sum_pair(const double* reg, int count) {
  double hi = 0.0, lo = 0.0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    hi = __dadd_rn(hi, reg[2 * i]);
    lo = __dadd_rn(lo, reg[2 * i + 1]);
  }
  __shared__ double sm[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const f64::HiLo w = f64::split(f64::warp_sum(hi));
  const double l = f64::value(f64::warp_sum(lo));
  if (lane == 0) {
    sm[warp] = w.hi;
    sm[16 + warp] = w.lo + l;
  }
  __syncthreads();
  f64::HiLo out{0.0, 0.0};
  if (warp == 0) out = f64::split(f64::warp_sum((lane & 15) < nw ? sm[lane] : 0.0));
  return out;
}
__device__ double region_sum_dd(const double* reg, int count) {
  const f64::HiLo w = region_sum_pair(reg, count);
  return w.hi + w.lo;
}

// beta and the invariants from the region sums rv, by warp 0
__device__ __forceinline__ void finish_step(const FinalizeArgs& a, const double* rv, double* out) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  // lane k: R[k] = <t_k, t_k+1> (k < 3), R[3] = <t_new, t_new>
  double Rk = 0.0;
  if (a.step) {
    const int re = lane < 3 ? R_IP_E + 2 * lane : R_44_E, rc = lane < 3 ? R_IP_C + 2 * lane : R_44_C;
    Rk = (rv[re] + rv[rc]) / a.totalArea;
  }
  double R[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) R[k] = __shfl_sync(0xffffffffu, Rk, k);
  if (threadIdx.x != 0) return;
  if (a.step) {
    double beta = 1.0;
    if (a.conserve) {
      if (a.scheme == 1)  // CRK3: R[0] = <t1,t2>, R[1] = <t1,t3>, R[2] = <t2,t3>
        beta = R[3] != 0.0 ? (2.0 * R[0] - R[1] + 2.0 * R[2]) / (3.0 * R[3]) : 1.0;
      else if (a.scheme == 3)  // PC2: R[0] = <t_old,t_new>, R[3] = <t_new,t_new>
        beta = (R[0] != 0.0 && R[3] != 0.0) ? R[0] / R[3] : 1.0;
      else  // CRK4
        beta = R[3] != 0.0 ? (R[0] + R[1] + R[2]) / (3.0 * R[3]) : 1.0;
      // time_scheme_mod.F90:145 (CRK4) and :94-100 (CRK3) divide 0 / 0 when the
      // tendency is zero everywhere (a state at rest); beta = 1 there, as the
      // reference's PC2 has it (:178)
    }
    out[4] = beta;
    out[5] = R[0];
    out[6] = R[1];
    out[7] = R[2];
    out[8] = R[3];
    out[9] = beta * a.dt;
  }
  if (a.diag) {
    out[0] = rv[R_MASS];
    out[1] = rv[R_EN_E] + rv[R_EN_C];
    out[2] = rv[R_PE];
    out[3] = rv[R_AV] / a.sumAreaTriangle;
  }
}

// a.split blocks per partial region (kFinSplit for one model, fewer for a
// batch of members), each the sum of a contiguous 1/a.split of the region's
// per-block partials into P.fin; the last block to finish (atomic counter, no
// waiting) combines each region's a.split sums (a warp per region) and the
// region sums into beta and the invariants (time_scheme_mod.F90:144-150;
// tmcore_swm_mod.F90:215-255), and re-arms the counter.  A thread adds its few
// blocks' sums in FP64, the lanes and warps are added as integers: with
// double-double shuffle trees on the 2-lane FP64 pipe this launch took 24 us at
// every mesh size; a level-6 FP32 step went from 118.3 to 102.8 us with the
// integer sums.
__global__ void __launch_bounds__(256) k_finalize(Partials P0, FinalizeArgs a, double* out0, double* res0,
                                                  unsigned int* counter0) {
  // one member per blockIdx.y: its partials, outputs, region sums and counter
  const Partials P = P0.at(blockIdx.y);
  double* out = out0 + (size_t)blockIdx.y * kDiagStride;
  double* res = res0 + (size_t)blockIdx.y * kDiagStride;
  unsigned int* counter = reinterpret_cast<unsigned int*>(reinterpret_cast<double*>(counter0) +
                                                          (size_t)blockIdx.y * kDiagStride);
  const int r = blockIdx.x / a.split, part = blockIdx.x - r * a.split;
  const bool want = (r <= R_44_E) ? a.step : a.diag;
  if (want) {
    const int count = a.counts[r], chunk = (count + a.split - 1) / a.split;
    const int i0 = min(count, part * chunk), i1 = min(count, i0 + chunk);
    const f64::HiLo v = region_sum_pair(P.region(r) + 2 * (size_t)i0, i1 - i0);
    if (threadIdx.x == 0) {
      P.fin[2 * (r * kFinSplit + part)] = v.hi;
      P.fin[2 * (r * kFinSplit + part) + 1] = v.lo;
    }
  }
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double rs[kFinalizeRegions];
  static_assert(2 * kFinSplit <= 32, "a warp combines one region's sums");
  const int lane = threadIdx.x & 31;
  for (int q = threadIdx.x >> 5; q < kFinalizeRegions; q += blockDim.x >> 5) {
    const bool on = ((q <= R_44_E) ? a.step : a.diag) && lane < 2 * a.split;
    // L2 loads: the other blocks wrote them
    const double s = f64::value(f64::warp_sum(on ? __ldcg(P.fin + 2 * q * kFinSplit + lane) : 0.0));
    if (lane == 0) rs[q] = res[q] = s;
  }
  __syncthreads();
  finish_step(a, rs, out);
  if (threadIdx.x == 0) *counter = 0u;
}

// The sum of `count` per-block pairs (their lo halves only if `lo`, else they are
// zero) by one warp, in every lane: up to 16 pairs per lane at a time, added
// exactly (f64::warp_sum).  A region has up to 30 pairs at level 5, 120 at 6, 480
// at 7; meshes with more than 512 add their rounds in double-double.  The terms
// go through a loop: this code runs once per step and region, and what counts is
// its fetch (16 pairs unrolled took a level-7 step 2.4 us, one unrolled form per
// number of pairs a level-6 step 1.9 us).
__device__ __forceinline__ double region_sum(const double* reg, int count, bool lo) {
  constexpr int K = 16;
  const int lane = threadIdx.x & 31;
  f64::HiLo sum{0.0, 0.0};
  for (int i0 = 0; i0 < count; i0 += 32 * K) {
    const int m = min(K, (count - i0 + 31) / 32);  // pairs of a lane
    double t[2 * K];
    for (int k0 = 0; k0 < m; k0 += 8)  // eight loads in flight
#pragma unroll
      for (int k = k0; k < k0 + 8; ++k) {
        const int i = i0 + 32 * k + lane;
        const double2 p = i < count ? __ldcg(reinterpret_cast<const double2*>(reg) + i) : make_double2(0.0, 0.0);
        t[lo ? 2 * k : k] = p.x;
        if (lo) t[2 * k + 1] = p.y;
      }
    const f64::HiLo r = f64::split(f64::warp_sum<1>(t, lo ? 2 * m : m));
    if (i0 == 0) {
      sum = r;
    } else {  // TwoSum (Knuth)
      const double h = __dadd_rn(sum.hi, r.hi), b = __dsub_rn(h, sum.hi);
      const double e = __dadd_rn(__dsub_rn(sum.hi, __dsub_rn(h, b)), __dsub_rn(r.hi, b));
      sum = {h, __dadd_rn(e, __dadd_rn(sum.lo, r.lo))};
    }
  }
  return sum.hi + sum.lo;
}

// The same after passes of one element per thread, for small FP32 models: the
// blocks first form the block sums those passes did not store, 256 threads of
// four elements with the fused multiply-adds, shuffle tree and block tree of
// the passes of kEPT elements per thread, so beta and the invariants do not
// depend on the passes' launch shapes; the last block to finish combines all
// regions, a warp each.
__device__ __forceinline__ void sum_products(const Partials& P, const float* f, const float* area, int n, int slot,
                                             const int (&r)[4]) {
  const int i0 = slot * (kEPT * 256) + threadIdx.x;
  float w[kEPT], x[4][kEPT], v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = 0; j < kEPT; ++j) {
    const int i = i0 + j * 256;
    w[j] = i < n ? area[i] : 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) x[k][j] = i < n ? f[(size_t)k * n + i] : 0.f;
  }
#pragma unroll
  for (int j = 0; j < kEPT; ++j)
    if (i0 + j * 256 < n)
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = __fmaf_rn(x[k][j], w[j], v[k]);
  block_store<float, 4>(v, P, r, slot);
}
__global__ void __launch_bounds__(256) k_finalize_products(Partials P, FinalizeArgs a, Products X, int nbc, int nbe,
                                                           int nbv, double* out, double* res, unsigned int* counter) {
  pdl_start();
  pdl_wait();
  const int b = blockIdx.x;
  if (b < nbc) {
    if (a.step) {
      const int r[4] = {R_IP_C, R_IP_C + 2, R_IP_C + 4, R_44_C};
      sum_products(P, X.c, X.areaCell_f, X.nc, b, r);
    }
    if (a.diag) {
      double mass = 0.0, enc = 0.0;
      float eh = 0.f, el = 0.f;
      for (int j = 0; j < kEPT; ++j) {
        const int i = b * (kEPT * 256) + j * 256 + threadIdx.x;
        if (i >= X.nc) break;
        const double g = X.gd[i], A = X.areaCell[i];
        mass = __fma_rn(g, A, mass);
        if (X.enc64) {
          enc = __fma_rn(g * __fma_rn(2.0, X.ghs[i], g), A, enc);
        } else {
          const float gf = X.gdf[i];
          two_sum_acc(eh, el, gf * (gf + 2.f * X.ghsf[i]) * X.areaCell_f[i]);
        }
      }
      const double v[2] = {mass, X.enc64 ? enc : (double)eh + (double)el};
      const int r[2] = {R_MASS, R_EN_C};
      block_store<double, 2>(v, P, r, b);
    }
  } else if (b < nbc + nbe) {
    const int slot = b - nbc;
    if (a.step) {
      const int r[4] = {R_IP_E, R_IP_E + 2, R_IP_E + 4, R_44_E};
      sum_products(P, X.e, X.areaEdge_f, X.ne, slot, r);
    }
    if (a.diag) {
      const bool ene64 = *X.en64 != 0;
      double en = 0.0;
      float eh = 0.f, el = 0.f;
      for (int j = 0; j < kEPT; ++j) {
        const int i = slot * (kEPT * 256) + j * 256 + threadIdx.x;
        if (i >= X.ne) break;
        const float t = X.iap[i] * X.iap[i] * X.areaEdge_f[i];
        if (ene64)
          en += (double)t;
        else
          two_sum_acc(eh, el, t);
      }
      const int r[1] = {R_EN_E};
      if (ene64) {
        const double v[1] = {en};
        block_store<double, 1>(v, P, r, slot);
      } else {
        const float h[1] = {eh}, l[1] = {el};
        block_store_ff<1>(h, l, P, r, slot);
      }
    }
  } else if (b < nbc + nbe + nbv) {
    const int slot = b - nbc - nbe;
    float ph = 0.f, pl = 0.f, ah = 0.f, al = 0.f;
    for (int j = 0; j < kEPT; ++j) {
      const int i = slot * (kEPT * 256) + j * 256 + threadIdx.x;
      if (i >= X.nv) break;
      two_sum_acc(ph, pl, X.v[i]);
      two_sum_acc(ah, al, X.v[(size_t)X.nv + i]);
      two_sum_acc(ah, al, X.fVertex_f[i] * X.areaTriangle_f[i]);
    }
    const float h[2] = {ph, ah}, l[2] = {pl, al};
    const int r[2] = {R_PE, R_AV};
    block_store_ff<2>(h, l, P, r, slot);
  }
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double rs[kFinalizeRegions];
  const int lane = threadIdx.x & 31;
  // warp w: the products' region w, whose block sums have no lo half, then an
  // invariant (in warps whose first region is the cells', a third of the edges)
  static_assert(R_44_E == 7 && kFinalizeRegions == 13, "eight warps, five invariants");
  constexpr unsigned kNone = 15, kSecond = (unsigned)R_EN_E | kNone << 4 | (unsigned)R_PE << 8 |
                                           (unsigned)R_EN_C << 12 | (unsigned)R_AV << 16 | kNone << 20 |
                                           (unsigned)R_MASS << 24 | kNone << 28;
  const unsigned warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int round = 0; round < 2; ++round) {
    const unsigned q = round ? kSecond >> (4 * warp) & 15u : warp;
    if (q == kNone) break;
    const int n = (round ? a.diag : a.step) ? a.counts[q] : 0;
    const double s = region_sum(P.region(q), n, round != 0);
    if (lane == 0) rs[q] = res[q] = s;
  }
  __syncthreads();
  finish_step(a, rs, out);
  if (threadIdx.x == 0) *counter = 0u;
}

void launch_finalize(Partials P, const int* counts_host, double totalArea, double sumAreaTriangle, double dt,
                     bool step, bool diag, bool conserve, double* diag_out, cudaStream_t st, int scheme,
                     int members, const Products* products, bool pdl) {
  FinalizeArgs a;
  for (int r = 0; r < R_COUNT; ++r) a.counts[r] = counts_host[r];
  a.totalArea = totalArea;
  a.sumAreaTriangle = sumAreaTriangle;
  a.dt = dt;
  a.step = step ? 1 : 0;
  a.diag = diag ? 1 : 0;
  a.conserve = conserve ? 1 : 0;
  a.scheme = scheme;
  // A single model's widest region (the edge partials of level 9: 15,360)
  // would leave one block's FP64 additions on one SM's 2-lane FP64 pipe, so
  // each region is split over kFinSplit blocks.  A batch of members already
  // has a block per region and member; splitting it as much multiplies the
  // blocks' fixed cost, so the split shrinks with the members (about
  // kFinSplit x the regions' blocks in all).
  const int nm = members > 1 ? members : 1;
  a.split = kFinSplit / nm > 1 ? kFinSplit / nm : 1;
  // scratch after the kDiagLen outputs: R_COUNT region sums, then the counter
  double* res = diag_out + kDiagLen;
  unsigned int* counter = reinterpret_cast<unsigned int*>(diag_out + kDiagLen + R_COUNT);
  if (products) {
    const int nbc = products->c ? grid_for(products->nc, 256) : 0, nbe = products->e ? grid_for(products->ne, 256) : 0;
    const int nbv = products->v && diag ? grid_for(products->nv, 256) : 0;
    launch(k_finalize_products, std::max(nbc + nbe + nbv, 1), Blk(256, 1, pdl), st, P, a, *products, nbc, nbe, nbv,
           diag_out, res, counter);
    return;
  }
  k_finalize<<<dim3(kFinalizeRegions * a.split, members > 1 ? members : 1), 256, 0, st>>>(P, a, diag_out, res,
                                                                                         counter);
}

// Conservative APVM epsilon (operators_mod.F90:349-354): one block per sum
// region R_C1..R_C3, the last block to finish computes
// eps = -(s1 - 2 s2) / (2 dt s3) into out[10] and re-arms its counter.
__global__ void __launch_bounds__(256) k_cons_eps(Partials P0, int count, double dt, double* out0, double* res0,
                                                  unsigned int* counter0) {
  const Partials P = P0.at(blockIdx.y);
  double* out = out0 + (size_t)blockIdx.y * kDiagStride;
  double* res = res0 + (size_t)blockIdx.y * kDiagStride;
  unsigned int* counter = reinterpret_cast<unsigned int*>(reinterpret_cast<double*>(counter0) +
                                                          (size_t)blockIdx.y * kDiagStride);
  const int r = R_C1 + blockIdx.x;
  const double v = region_sum_dd(P.region(r), count);
  if (threadIdx.x == 0) res[r] = v;
  __shared__ bool last;
  if (threadIdx.x == 0) {
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  volatile const double* rv = res;
  const double s1 = rv[R_C1], s2 = rv[R_C2], s3 = rv[R_C3];
  // eps = 0 when s3 = 0: with no wind the correction dpv is zero on every
  // edge and the reference's quotient is 0 / 0 (operators_mod.F90:349-351)
  out[10] = s3 != 0.0 ? -(s1 - s2 * 2.0) / (2.0 * dt * s3) : 0.0;
  *counter = 0u;
}

void launch_cons_eps(Partials P, int count, double dt, double* diag_out, cudaStream_t st, int members) {
  double* res = diag_out + kDiagLen;
  unsigned int* counter = reinterpret_cast<unsigned int*>(diag_out + kDiagLen + R_COUNT + 1);
  k_cons_eps<<<dim3(3, members > 1 ? members : 1), 256, 0, st>>>(P, count, dt, diag_out, res, counter);
}

// adv model spatial operator, edges: c2e + upwind correction with the sign of
// u (operators_mod.F90:93-104, :423-472), mass flux u*gd_edge
// (adv_scheme_sg11_mod.F90:42-46)
__global__ void __launch_bounds__(kMaxBlock) k_adv_edge(DevMesh M, ModelOpt O, const double* gd, const double* u,
                                                        double* gd_e, double* F) {
  TMC_FOR_EPT(e, M.ne) {
    const int c1 = M.cellsOnEdge[e], c2 = M.cellsOnEdge[M.ne + e];
    const double ue = u[e];
    double ge = 0.5 * (gd[c1] + gd[c2]);
    if (O.adv_order >= 3)
      ge = upwind_edge<double>(M.cell2, M.cell4, O.adv_order, O.cell_coef2, O.cell_coef4, M.ne, e, c1, c2, ge, ue,
                               M.dcEdge[e], [gd](int i) { return gd[i]; });
    gd_e[e] = ge;
    F[e] = ue * ge;
  }
}

// div_operator (operators_mod.F90:40-55) of the mass flux
__global__ void __launch_bounds__(kMaxBlock) k_adv_div(DevMesh M, const double* F, double* tend) {
  TMC_FOR_EPT(c, M.nc) {
    double s = 0.0;
    for (int i = 0; i < M.nEdgesOnCell[c]; ++i) {
      const int e = M.edgesOnCell[(size_t)i * M.nc + c];
      s = s + (double)M.nSign[(size_t)i * M.nc + c] * F[e] * M.dvEdge[e];
    }
    tend[c] = (-s) / M.areaCell[c];
  }
}

void launch_adv_spatial(const DevMesh& M, const ModelOpt& O, const double* gd, const double* u, double* gd_e,
                        double* F, double* tend, int bs, cudaStream_t st) {
  k_adv_edge<<<grid_for(M.ne, bs), bs, 0, st>>>(M, O, gd, u, gd_e, F);
  k_adv_div<<<grid_for(M.nc, bs), bs, 0, st>>>(M, F, tend);
}

// stream function of the prescribed wind on vertices
__global__ void k_adv_psi(int nv, int wind_case, double radius, const double* latV, const double* lonV,
                          const double* t0, double offset, const double* offset_dev, double* psi) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const double pi = 4.0 * atan(1.0);
  const double lat = latV[v], lon = lonV[v];
  if (wind_case == 1) {
    // cosine_bell_rotation_test_mod.F90:45-68 (alpha = pi/2, one revolution in 12 days)
    const double u0 = 2.0 * pi * radius / 12.0 / 86400.0, alpha = 0.5 * pi;
    const double ca = cos(alpha), sa = sin(alpha);
    psi[v] = -radius * u0 * (sin(lat) * ca - cos(lon) * cos(lat) * sa);
  } else {
    // deformation_flow_test_mod.F90:74-105 (case 4: deformation plus solid-body rotation)
    const double seconds = *t0 + (offset_dev ? *offset_dev : offset);
    const double T0 = 12.0 * 86400.0, u0 = 2.0 * pi * radius / T0;
    const double c = pi * 2.0 * seconds / T0, k = 10.0 * radius / T0, cosT = cos(pi * seconds / T0);
    const double sn = sin(lon - c), cl = cos(lat);
    const double p = k * (sn * sn) * (cl * cl) * cosT - u0 * sin(lat);
    psi[v] = p * radius;
  }
}

__global__ void k_adv_u(int ne, const int32_t* verticesOnEdge, const double* dvEdge, const double* psi, double* u) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= ne) return;
  u[e] = -(psi[verticesOnEdge[ne + e]] - psi[verticesOnEdge[e]]) / dvEdge[e];
}

void launch_adv_wind(const DevMesh& M, int wind_case, double radius, const double* latV, const double* lonV,
                     const double* t0_dev, double offset, const double* offset_dev, double* psi, double* u,
                     cudaStream_t st) {
  k_adv_psi<<<nblk(M.nv, 256), 256, 0, st>>>(M.nv, wind_case, radius, latV, lonV, t0_dev, offset, offset_dev, psi);
  k_adv_u<<<nblk(M.ne, 256), 256, 0, st>>>(M.ne, M.verticesOnEdge, M.dvEdge, psi, u);
}

__global__ void k_adv_advance(double* elapsed, double dt) { *elapsed = *elapsed + dt; }

void launch_adv_advance(double* elapsed_dev, double dt, cudaStream_t st) {
  k_adv_advance<<<1, 1, 0, st>>>(elapsed_dev, dt);
}

// total mass (tmcore_swm_mod.F90:215-220) alone; the other invariant regions
// get zero partials so that the finaliser reports 0 for them
__global__ void __launch_bounds__(kMaxBlock) k_mass_only(DevMesh M, const double* gd, Partials P) {
  double mass = 0.0;
  TMC_FOR_EPT(c, M.nc) mass = mass + gd[c] * M.areaCell[c];
  const double v[5] = {mass, 0.0, 0.0, 0.0, 0.0};
  const int r[5] = {R_MASS, R_EN_E, R_EN_C, R_PE, R_AV};
  block_store<double, 5>(v, P, r);
}

int launch_mass_only(const DevMesh& M, const double* gd, Partials P, int bs, cudaStream_t st) {
  const int g = grid_for(M.nc, bs);
  k_mass_only<<<g, bs, 0, st>>>(M, gd, P);
  return g;
}

// h = (gd + ghs) / g (history_mod.F90:166)
__global__ void k_h_field(int nc, const double* gd, const double* ghs, double g, double* h) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nc) h[c] = (gd[c] + ghs[c]) / g;
}

void launch_h_field(int nc, const double* gd, const double* ghs, double g, double* h, cudaStream_t st) {
  k_h_field<<<nblk(nc, 256), 256, 0, st>>>(nc, gd, ghs, g, h);
}

// gdf = FP32 gd (skipped when null), qr = q / FP32 gd
__global__ void k_shadows(int nc, int ntr, const double* gd, const float* q, float* gdf, float* qr) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nc) return;
  const float g = (float)gd[c];
  if (gdf) gdf[c] = g;
  for (int k = 0; k < ntr; ++k) qr[(size_t)k * nc + c] = q[(size_t)k * nc + c] / g;
}

void launch_shadows(int nc, int ntr, const double* gd, const float* q, float* gdf, float* qr, cudaStream_t st) {
  k_shadows<<<nblk(nc, 256), 256, 0, st>>>(nc, ntr, gd, q, gdf, qr);
}

__global__ void k_to_f32(size_t n, const double* src, float* dst) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (float)src[i];
}

void launch_to_f32(size_t n, const double* src, float* dst, cudaStream_t st) {
  k_to_f32<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, src, dst);
}

// ---------------------------------------------------------------------------
// single operators (operators_mod.F90), FP64, reference expression order
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kMaxBlock) k_op(int op, DevMesh M, const double* a, const double* b,
                                                  const double* c, double* out, int order, double coef2,
                                                  double coef4) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  switch (op) {
    case OP_DIV:  // :40-55
      if (i < M.nc) {
        double s = 0.0;
        for (int k = 0; k < M.nEdgesOnCell[i]; ++k) {
          int e = M.edgesOnCell[(size_t)k * M.nc + i];
          s = s + (double)M.nSign[(size_t)k * M.nc + i] * a[e] * M.dvEdge[e];
        }
        out[i] = (-s) / M.areaCell[i];
      }
      break;
    case OP_CURL:  // :76-91
      if (i < M.nv) {
        double s = 0.0;
        for (int k = 0; k < 3; ++k) {
          int e = M.edgesOnVertex[(size_t)k * M.nv + i];
          s = s + (double)M.tSign[(size_t)k * M.nv + i] * a[e] * M.dcEdge[e];
        }
        out[i] = (-s) / M.areaTriangle[i];
      }
      break;
    case OP_C2E:  // :93-104
      if (i < M.ne) out[i] = 0.5 * (a[M.cellsOnEdge[i]] + a[M.cellsOnEdge[M.ne + i]]);
      break;
    case OP_C2V:  // :106-123
      if (i < M.nv) {
        double s = 0.0;
        for (int k = 0; k < 3; ++k) s = s + a[M.cellsOnVertex[(size_t)k * M.nv + i]] * M.kite[(size_t)k * M.nv + i];
        out[i] = s / M.areaTriangle[i];
      }
      break;
    case OP_V2C:  // :125-141
      if (i < M.nc) {
        double s = 0.0;
        for (int k = M.v2c_start[i]; k < M.v2c_start[i + 1]; ++k)
          s = s + a[M.v2c_vertex[k]] * M.v2c_kite[k] / M.areaCell[i];
        out[i] = s;
      }
      break;
    case OP_V2E:  // :143-156
      if (i < M.ne) out[i] = 0.5 * (a[M.verticesOnEdge[i]] + a[M.verticesOnEdge[M.ne + i]]);
      break;
    case OP_KE:  // :206-221
      if (i < M.nc) {
        double s = 0.0;
        for (int k = 0; k < M.nEdgesOnCell[i]; ++k) {
          int e = M.edgesOnCell[(size_t)k * M.nc + i];
          s = s + a[e] * a[e] * M.areaEdge[e];
        }
        out[i] = (s * 0.25) / M.areaCell[i];
      }
      break;
    case OP_TWIND:  // :223-237
      if (i < M.ne) {
        double s = 0.0;
        for (int k = 0; k < M.nEdgesOnEdge[i]; ++k)
          s = s + a[M.edgesOnEdge[(size_t)k * M.ne + i]] * M.weightsOnEdge[(size_t)k * M.ne + i];
        out[i] = s;
      }
      break;
    case OP_TVF:  // :239-260
      if (i < M.ne) {
        double s = 0.0;
        for (int k = 0; k < M.nEdgesOnEdge[i]; ++k) {
          int ep = M.edgesOnEdge[(size_t)k * M.ne + i];
          s = s + M.weightsOnEdge[(size_t)k * M.ne + i] * a[ep] * b[ep] * 0.5 * (c[i] + c[ep]);
        }
        out[i] = s;
      }
      break;
    case OP_UPWIND:  // :423-472
      if (i < M.ne) {
        const int c1 = M.cellsOnEdge[i], c2 = M.cellsOnEdge[M.ne + i];
        out[i] = upwind_edge<double>(M.cell2, M.cell4, order, coef2, coef4, M.ne, i, c1, c2, out[i], b[i],
                                     M.dcEdge[i], [a](int j) { return a[j]; });
      }
      break;
  }
}

void launch_op(int op, const DevMesh& M, const ModelOpt& O, const double* a, const double* b, const double* c,
               double* out, int order, int mono, double coef2, double coef4, int bs, cudaStream_t st) {
  (void)O;
  (void)mono;
  int n = M.ne;
  if (op == OP_DIV || op == OP_V2C || op == OP_KE) n = M.nc;
  if (op == OP_CURL || op == OP_C2V) n = M.nv;
  k_op<<<nblk(n, bs), bs, 0, st>>>(op, M, a, b, c, out, order, coef2, coef4);
}

}  // namespace tmc
