#pragma once

#include <stdint.h>

namespace akb {

// prescribed velocity ramp on a list of dofs (u indices node * D + c): step k
// sets them to u0 + acc, acc growing by dt v_max min(1, k / ramp) per step;
// acc and the step count live on the device.  Bit kPrescribedBit + c of a
// node's blocked flags marks its component c as such a dof.
constexpr int kPrescribedBit = 4;
struct PrescArgs {
  int64_t count = 0;  // 0: none
  const int64_t *dofs = nullptr;
  const double *u0 = nullptr;
  double v_max = 0., ramp = 1., dt = 0.;
  double *acc = nullptr;
  int64_t *step = nullptr;
};

}  // namespace akb
