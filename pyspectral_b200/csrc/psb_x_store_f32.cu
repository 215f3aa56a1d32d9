// Register x pass and epilogue, float fields: product spectra stored as they are.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(float, EpiStore<float, 6>)
PSB_REG_X_OF(float, EpiStore<float, 9>)
PSB_REG_X_OF(float, EpiStore<float, 12>)
}  // namespace psbh
