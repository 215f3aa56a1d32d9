// Register x pass and epilogue, double fields: the memory models' two stages.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(double, EpiPL<double>)
PSB_REG_X_OF(double, EpiPLQL<double>)
}  // namespace psbh
