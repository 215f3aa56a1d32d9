// Register x pass and epilogue, float fields: MHD and its t-model.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(float, EpiMHD<float>)
PSB_REG_X_OF(float, EpiMHDQ<float>)
PSB_REG_X_OF(float, EpiMHDT<float>)
}  // namespace psbh
