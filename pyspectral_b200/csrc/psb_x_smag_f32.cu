// Register x pass and epilogue, float fields: Smagorinsky stages.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(float, EpiSmagStep<float>)
PSB_REG_X_BATCH_OF(float, EpiSmagStep<float>)
}  // namespace psbh
