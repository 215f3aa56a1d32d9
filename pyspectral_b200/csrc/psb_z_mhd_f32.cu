// Register z pass, float fields: MHD products and their linearisation.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(float, PhysMHD<float>)
PSB_REG_Z(float, PhysMHDLin<float>)
}  // namespace psbh
