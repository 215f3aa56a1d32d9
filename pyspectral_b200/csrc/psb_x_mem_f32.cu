// Register x pass and epilogue, float fields: the memory models' two stages.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(float, EpiPL<float>)
PSB_REG_X_OF(float, EpiPLQL<float>)
}  // namespace psbh
