// Register x pass and epilogue, double fields: Smagorinsky stages.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(double, EpiSmagStep<double>)
PSB_REG_X_BATCH_OF(double, EpiSmagStep<double>)
}  // namespace psbh
