// Register z pass, double fields: products and the Smagorinsky stress.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(double, PhysSmag<double>)
PSB_REG_Z_BATCH(double, PhysSmag<double>)
}  // namespace psbh
