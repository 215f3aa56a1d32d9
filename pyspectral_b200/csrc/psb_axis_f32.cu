// Register axis passes, float fields.
#include "psb_axis.cuh"

namespace psbh {
template int reg_axis<float>(psb_ctx*, const psb::AxisArgs<float>&, const psb::FieldTab<float>&, bool, const char*, double);
template int reg_axis_batch<float>(psb_ctx*, const psb::AxisArgs<float>*, const psb::FieldTab<float>&, int, int, int, int,
                                  bool, const char*, double);
}  // namespace psbh
