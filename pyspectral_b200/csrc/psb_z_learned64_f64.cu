// Register z pass, double fields: products and the learned stress, width-64 network.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(double, PhysLearned<double, kActRelu, 64>)
PSB_REG_Z_BATCH(double, PhysLearned<double, kActRelu, 64>)
}  // namespace psbh
