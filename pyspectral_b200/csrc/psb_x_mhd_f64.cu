// Register x pass and epilogue, double fields: MHD and its t-model.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(double, EpiMHD<double>)
PSB_REG_X_OF(double, EpiMHDQ<double>)
PSB_REG_X_OF(double, EpiMHDT<double>)
}  // namespace psbh
