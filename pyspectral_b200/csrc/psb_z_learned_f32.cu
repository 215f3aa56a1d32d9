// Register z pass, float fields: products and the learned stress, width-32 network.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(float, PhysLearned<float, kActRelu, 32>)
PSB_REG_Z_BATCH(float, PhysLearned<float, kActRelu, 32>)
}  // namespace psbh
