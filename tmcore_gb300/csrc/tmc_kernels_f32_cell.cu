// FP32 instantiation of the cell passes (tmc_kernels_f32.cu has the others), and
// a small model's cell and vertex pass of a stage in one launch: blocks [0, nvb)
// take the vertices, the others the cells.
#include "tmc_kernels_impl.cuh"

namespace tmc {

TMC_INSTANTIATE_CELL(float)

namespace {

__global__ void __launch_bounds__(kMaxBlock) k_cell_vertex(DevMesh M, ModelOpt O, StageIO<float> S, RKStage rk,
                                                           Partials P, int diag, int nvb) {
  if ((int)blockIdx.x < nvb)
    vertex_body<float, false, 1, true>(M, S, P, diag);
  else
    cell_body<float, false, 1, true>(M, O, S, rk, P, diag, nvb);
}
template <int NTR, int kMode>
__global__ void __launch_bounds__(kCellBlock, TMC_CELL_SINGLE_MIN_BLOCKS)
    k_cell_vertex_fast(DevMesh M, StageIO<float> S, RKStage rk, Partials P, int diag, int nvb) {
  if ((int)blockIdx.x < nvb)
    vertex_body<float, false, 1, true>(M, S, P, diag);
  else
    cell_fast_body<NTR, false, 1, kMode, true>(M, S, rk, P, diag, nvb);
}

}  // namespace

void launch_cell_vertex(const DevMesh& M, const ModelOpt& O, const StageIO<float>& S, RKStage rk, Partials P, bool diag,
                        Blk b, cudaStream_t st) {
  const int nvb = grid_for(M.nv, b), g = nvb + grid_for(M.nc, b), dg = diag ? 1 : 0;
  auto run = [&](auto ntr) {
    on_mode(!S.gd_e, rk.mode, [&](auto m) {
      constexpr int kMode = decltype(m)::value;
      if constexpr (kMode != 0)
        launch(k_cell_vertex_fast<decltype(ntr)::value, kMode>, g, b, st, M, S, rk, P, dg, nvb);
    });
  };
  if (launch_cell_is_fast(O)) {
    switch (O.n_tracers) {
      case 0: run(std::integral_constant<int, 0>()); return;
      case 1: run(std::integral_constant<int, 1>()); return;
      case 2: run(std::integral_constant<int, 2>()); return;
      case 4: run(std::integral_constant<int, 4>()); return;
      default: break;
    }
  }
  launch(k_cell_vertex, g, b, st, M, O, S, rk, P, dg, nvb);
}

}  // namespace tmc
