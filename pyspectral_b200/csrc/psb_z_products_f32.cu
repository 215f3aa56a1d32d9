// Register z pass, float fields: products of the velocity (DNS, the memory models' first stage).
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(float, PhysProducts<float>)
PSB_REG_Z_BATCH(float, PhysProducts<float>)
}  // namespace psbh
