// train_ctl.h -- what a training epoch leaves beside its parameters (kappa.cu).
#pragma once

namespace imcom {

struct TrainCtl {
  float loss;        // summed over the epoch
  unsigned arrived;  // the grid barrier's count
  int err;           // not zero: the barrier timed out
  int pad;
};
static_assert(sizeof(TrainCtl) == 16, "four words per epoch");

// Whether any epoch's barrier timed out (whole numbers, so the caller's treatment of
// denormals does not matter).
inline bool train_failed(const TrainCtl* ctl, int epochs) {
  for (int ep = 0; ep < epochs; ++ep)
    if (ctl[ep].err != 0) return true;
  return false;
}

}  // namespace imcom
