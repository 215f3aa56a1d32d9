// Register z pass, double fields: products of the velocity (DNS, the memory models' first stage).
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(double, PhysProducts<double>)
PSB_REG_Z_BATCH(double, PhysProducts<double>)
}  // namespace psbh
