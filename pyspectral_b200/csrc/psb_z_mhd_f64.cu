// Register z pass, double fields: MHD products and their linearisation.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(double, PhysMHD<double>)
PSB_REG_Z(double, PhysMHDLin<double>)
}  // namespace psbh
