// Register z pass, float fields: products of the velocity and the unresolved rate of change.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(float, PhysPLQL<float>)
PSB_REG_Z(float, PhysPLQS<float>)
}  // namespace psbh
