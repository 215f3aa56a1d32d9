// Register z pass, double fields: products and the learned stress, width-32 network.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(double, PhysLearned<double, kActRelu, 32>)
PSB_REG_Z_BATCH(double, PhysLearned<double, kActRelu, 32>)
}  // namespace psbh
