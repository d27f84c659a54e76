// The windowed back-projection over plain detector rows: windows of 4-byte pixels,
// half the shared memory of row pairs and boxes of up to 256 columns, for axes whose
// row pairs leave too few CTAs on an SM or fit no box (several detector pixels per
// voxel).  Separate from bp_tma.cu so that the instantiations compile in parallel.
#include "bp_brick.cuh"

namespace mtr {

namespace {
template <int MODE, int LANES>
cudaError_t launch_bz(const CUtensorMap& map, const BpArgs& P, const BpPlan& plan, cudaStream_t st) {
  return plan.bz0 ? launch_nz<float, MODE, false, LANES, true, 3>(map, P, plan, st)
                  : launch_nz<float, MODE, false, LANES, false, 3>(map, P, plan, st);
}
template <int MODE>
cudaError_t launch_lanes(const CUtensorMap& map, const BpArgs& P, const BpPlan& plan, cudaStream_t st) {
  return plan.lanes == 2 ? launch_bz<MODE, 2>(map, P, plan, st) : plan.lanes == 1 ? launch_bz<MODE, 1>(map, P, plan, st)
                                                                                  : launch_bz<MODE, 0>(map, P, plan, st);
}
}  // namespace

cudaError_t launch_backproject_tma_rows(const CUtensorMap& map, const BpPlan& plan, const BpArgs& P,
                                        cudaStream_t st) {
  return P.mode == 0 ? launch_lanes<0>(map, P, plan, st) : launch_lanes<1>(map, P, plan, st);
}

}  // namespace mtr
