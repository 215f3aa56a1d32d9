// Host side of the register axis passes (psb_reg.cuh): one translation unit
// per precision instantiates every length.
#pragma once
#include "psb_ctx.cuh"
#include "psb_reg.cuh"

namespace psbh {

template <typename T, int A, int B, bool INV>
int launch_reg_axis(psb_ctx* c, const psb::AxisArgs<T>& a, const psb::FieldTab<T>& ft, const char* what,
                    double bytes) {
  constexpr int C = psb::reg_cols<T>();
  constexpr size_t smem = (size_t)A * B * C * sizeof(Cx<T>);
  set_smem(psb::axis_reg_kernel<T, A, B, INV>, smem);
  LaunchScope scope(c, what, bytes);
  const dim3 grid((a.ncols + C - 1) / C, a.nouter, ft.nf);
  const bool serial = serial_after_z(scope.after_z, (long long)grid.x * grid.y * grid.z, 148LL * psb::axis_reg_minb<T, A>());
  launch_pdl_if(!serial, psb::axis_reg_kernel<T, A, B, INV>, grid, A * C, smem, c->stream, a, ft);
  return launch_ok(c, what);
}

template <typename T>
int reg_axis(psb_ctx* c, const psb::AxisArgs<T>& a, const psb::FieldTab<T>& ft, bool inv, const char* what,
             double bytes) {
  switch (a.plan.L) {
#define PSB_CASE(L, A, B)                                                               \
  case L:                                                                               \
    return inv ? launch_reg_axis<T, A, B, true>(c, a, ft, what, bytes)                  \
               : launch_reg_axis<T, A, B, false>(c, a, ft, what, bytes);
    PSB_REG_AXIS(PSB_CASE)
#undef PSB_CASE
    default:
      return fail(c, PSB_ERR_SHAPE, std::string(what) + ": no register pass of this length");
  }
}

template <typename T, int A, int B, bool INV>
int launch_reg_axis_batch(psb_ctx* c, const psb::AxisArgs<T>* args, const psb::FieldTab<T>& ft, int ncols, int nouter,
                          int runs, const char* what, double bytes) {
  constexpr int C = psb::reg_cols<T>();
  constexpr size_t smem = (size_t)A * B * C * sizeof(Cx<T>);
  set_smem(psb::axis_reg_batch<T, A, B, INV>, smem);
  LaunchScope scope(c, what, bytes);
  const dim3 grid((ncols + C - 1) / C * runs, nouter, ft.nf);
  const bool serial = serial_after_z(scope.after_z, (long long)grid.x * grid.y * grid.z, 148LL * psb::axis_reg_minb<T, A>());
  launch_pdl_if(!serial, psb::axis_reg_batch<T, A, B, INV>, grid, A * C, smem, c->stream, args, ft);
  return launch_ok(c, what);
}

template <typename T>
int reg_axis_batch(psb_ctx* c, const psb::AxisArgs<T>* args, const psb::FieldTab<T>& ft, int L, int ncols, int nouter,
                   int runs, bool inv, const char* what, double bytes) {
  switch (L) {
#define PSB_CASE(LEN, A, B)                                                                                    \
  case LEN:                                                                                                    \
    return inv ? launch_reg_axis_batch<T, A, B, true>(c, args, ft, ncols, nouter, runs, what, bytes)           \
               : launch_reg_axis_batch<T, A, B, false>(c, args, ft, ncols, nouter, runs, what, bytes);
    PSB_REG_AXIS(PSB_CASE)
#undef PSB_CASE
    default:
      return fail(c, PSB_ERR_SHAPE, std::string(what) + ": no register pass of this length");
  }
}

}  // namespace psbh
