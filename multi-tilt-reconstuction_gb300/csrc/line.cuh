// Projector pair for tilt axes whose detector x does not move along one volume
// axis (single-axis tomography with the tilt axis along Y or X, and each axis
// of a dual-axis series): declarations shared with the reconstruction.
//
// Such a geometry separates.  With w the volume axis that detector x ignores
// (the lines) and m the other in-plane axis,
//     x = a0 + am m + a3 z - 1,     y = b0 + bw w - 1,
// so every line of voxels along w meets the same two detector columns with the
// same weights, and the interpolation along y involves w alone.  The kernels
// therefore work on line images [angle][x][w]: the projections resampled onto
// the volume's own w positions (detector row interpolation done once per
// angle, x and w instead of once per voxel), or, going forward, line sums that
// are spread over the detector rows once.  With the lanes of a warp along w
// the x position, its fraction and every pixel crossing are the same for all
// 32 lanes: no divergence, no bank conflicts, and the scalar work is shared by
// the 2 or 4 values a lane holds.
#pragma once

#include "mtr_internal.h"

namespace mtr {

struct LinePlan {
  bool ok = false;
  int along_x = 0;        // lines along X (else along Y)
  int W = 0, Wp = 0;      // line length and pitch of a line image's rows
  int fwd_vl = 4, fwd_nz = 16, fwd_rows = 0;  // forward: values per lane, depth, window rows
  int bp_vl = 4, bp_nz = 8, bp_rows = 0;     // SIRT update
  int wbp_vl = 4, wbp_nz = 8, wbp_rows = 0;   // WBP
  int n_tab = 1;          // angles in the row tables (1: the same y-map at every angle)
  // row tables (host), uploaded by the reconstruction as one array:
  // [n_tab][Wp] {row below, fraction}, [n_tab][PY] {first line position, count},
  // [n_tab][Wp] weight on the detector
  std::vector<int> tables;
  size_t off_rows = 0, off_weight = 0;  // words
};

// Lines along X or Y when every map of the axis separates (to 1e-6 px over
// the volume) and the line images fit the axis' projection-space arrays;
// depth: planes of one launch.
LinePlan plan_lines(const std::vector<double>& xc, const std::vector<double>& yc, int A, int PX, int PY, int pitch,
                    const VolDev& vol, int depth, int sms);

// The tables on the device.
struct LineTab {
  const int2* row = nullptr;      // [n_tab][Wp]
  const int2* span = nullptr;     // [n_tab][PY]
  const float* weight = nullptr;  // [n_tab][Wp]
  int stride = 0;                 // tables per angle: 0 when shared
};

// Line sums of the volume planes [z0, z1) (x null: of ones) added into the
// line image behind `map` ([A][PX][W], box W: 32 * fwd_vl by fwd_rows).
template <typename VT>
cudaError_t launch_line_forward(const CUtensorMap& map, const LinePlan& p, const AxisDev& ax, const VolDev& vol,
                                const VT* x, int z0, int z1, cudaStream_t st);
// mode 0 WBP, 1 SIRT update, over the line image behind `map`.
cudaError_t launch_line_backproject(const CUtensorMap& map, const LinePlan& p, const LineTab& tab, const AxisDev& ax,
                                    const VolDev& vol, int mode, float step, float* vol_out, float* cbp,
                                    void* vol_copy, int copy_kind, int z0, int z1, int* err, cudaStream_t st);
// Between the two spaces, per angle and detector column:
//   mode 0: s = line sums spread over the rows; residual b - s/cf; written as
//           a line image to `image`; the line sums reset to zero; norm2 (or
//           null) accumulates the squared residual in FP64
//   mode 1: cf = line sums spread over the rows; the line sums reset to zero
//   mode 2: b as a line image
template <typename BT>
cudaError_t launch_line_rows(int mode, const LinePlan& p, const LineTab& tab, const AxisDev& ax, const BT* b,
                             float* sums, float* cf, float* image, double* norm2, cudaStream_t st);

}  // namespace mtr
