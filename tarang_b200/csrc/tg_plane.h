// y-inverse, z-pass and y-forward of a small x-plane in one kernel (tg_plane.cu).
#pragma once

#include "tg_fft_launch.h"

namespace tg {

struct PlaneArgs {
  AxisMap ay;           // stored rows of the y axis
  int nky, kzp, nkz;    // stored rows, row length and entries in use of a row of both sides
  int rin, rout;        // row strides in shared memory (complex elements) of inputs and products
  unsigned mkz, mkzp;   // reciprocals of nkz and kzp
  int nin, nprod;
  double scale;
  const cx<double>* twy;  // exp(-2 pi i m / N2)
  const cx<double>* twN;  // exp(-2 pi i m / N3)
};

struct PlaneLaunch {
  int N2 = 0, M = 0;    // M = N3/2
  int prec = F64;
  long long nplanes = 0;  // requests x N1
  PlaneArgs a{};          // rin .. mkzp are set by the launcher
  PtrSet ps{};            // src: x-inverse outputs [N1][nky][kzp], dst: y-forward outputs, alike
  ProdPairs pp{};
};

// whether the planes of a grid with N1 of them are taken by launch_plane
bool plane_fits(const PlaneLaunch& l, int N1);
cudaError_t launch_plane(PlaneLaunch l, cudaStream_t s);

}  // namespace tg
