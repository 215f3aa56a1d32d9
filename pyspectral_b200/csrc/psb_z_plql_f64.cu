// Register z pass, double fields: products of the velocity and the unresolved rate of change.
#include "psb_z.cuh"

namespace psbh {
using namespace psb;
PSB_REG_Z(double, PhysPLQL<double>)
PSB_REG_Z(double, PhysPLQS<double>)
}  // namespace psbh
