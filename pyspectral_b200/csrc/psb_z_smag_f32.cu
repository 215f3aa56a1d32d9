// Register z pass, float fields: products and the Smagorinsky stress.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(float, PhysSmag<float>)
PSB_REG_Z_BATCH(float, PhysSmag<float>)
}  // namespace psbh
