// Register x pass and epilogue, double fields: Navier-Stokes, and Smagorinsky with its closure force.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(double, EpiNS<double, false>)
PSB_REG_X_BATCH_OF(double, EpiNS<double, false>)
PSB_REG_X_OF(double, EpiNS<double, true>)
}  // namespace psbh
