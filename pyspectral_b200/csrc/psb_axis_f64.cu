// Register axis passes, double fields.
#include "psb_axis.cuh"

namespace psbh {
template int reg_axis<double>(psb_ctx*, const psb::AxisArgs<double>&, const psb::FieldTab<double>&, bool, const char*, double);
template int reg_axis_batch<double>(psb_ctx*, const psb::AxisArgs<double>*, const psb::FieldTab<double>&, int, int, int, int,
                                  bool, const char*, double);
}  // namespace psbh
