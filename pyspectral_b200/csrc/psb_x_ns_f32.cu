// Register x pass and epilogue, float fields: Navier-Stokes, and Smagorinsky with its closure force.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(float, EpiNS<float, false>)
PSB_REG_X_BATCH_OF(float, EpiNS<float, false>)
PSB_REG_X_OF(float, EpiNS<float, true>)
}  // namespace psbh
