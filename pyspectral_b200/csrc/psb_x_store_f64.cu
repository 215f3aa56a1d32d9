// Register x pass and epilogue, double fields: product spectra stored as they are.
#include "psb_x.cuh"

namespace psbh {
using namespace psb;
PSB_REG_X_OF(double, EpiStore<double, 6>)
PSB_REG_X_OF(double, EpiStore<double, 9>)
PSB_REG_X_OF(double, EpiStore<double, 12>)
}  // namespace psbh
