// The x-forward pass, an RK stage and the next x-inverse in one kernel (tg_xstage.cu).
#pragma once

#include "tg_fft_launch.h"
#include "tg_spectral.cuh"

namespace tg {

struct XStageLaunch {
  int phys = 0;             // PH_FLUID, PH_MHD, PH_SCALAR
  int prec = F64;           // transform precision
  RKArgs rk{};              // stage 1, 2, 3 or 7; PX is not used
  int us_all = 0;           // write every stage value to US (else those inside the force box)
  const cx<double>* tw = nullptr;  // exp(-2 pi i m / N1)
  int* wait_flag = nullptr;
  int wait_short = 0;
  const void* src[8] = {};  // y-forward outputs [N1][nky][kzp] of the trace-free products
  void* dst[6] = {};        // x-inverse outputs [N1][nky][kzp]
};

// whether a step of nact requests on this grid runs its non-final stages through launch_xstage (FOUR, N1 of
// 32 .. 256)
bool xstage_fits(const Geo& g, int phys, int prec, int nact);
cudaError_t launch_xstage(const XStageLaunch& l, cudaStream_t s, bool* used);

}  // namespace tg
