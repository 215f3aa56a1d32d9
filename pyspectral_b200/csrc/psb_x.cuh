// Host side of the register x pass (psb_xreg.cuh); the psb_x_*.cu translation
// units instantiate it for a set of epilogues and one precision each.
#pragma once
#include "psb_ctx.cuh"

namespace psbh {

// Blocks of nt threads for the columns without products: one mode a thread.
inline int x_extra_blocks(int n1, int n2, int ncz, int nt) {
  const long long pts = (long long)n1 * n2 * ncz;
  return (int)std::min<long long>((pts + nt - 1) / nt, 4096);
}

// Blocks up to which a launch takes three groups of threads a tile: every CTA is
// resident at once (FP32 Smagorinsky 48^3 14.6 us against 22.8 with one group,
// learned 36^3 10.2 against 12.3); beyond that the groups only take CTAs from an SM
// that has more to run.  0: never.  FP64 launches this small run the staged pass
// (x_pass_in_registers), and a block of three groups has at most 1024 threads.
template <typename T, class Epi, int A, int B, int R>
constexpr int x_group_wave() {
  if (sizeof(T) == 8 || Epi::NACC == 0 || 3 * psb::xreg_threads<T, A, B>() > 1024) return 0;
  return 148 * (psb::xreg_minb<T, Epi, A, B, R, true>() / 3);
}

template <typename T, class Epi, int A, int B, int R, int S, bool MANY>
int launch_reg_xs(psb_ctx* c, const psb::XEpiArgs<T>& e, const Epi& epi, const char* what, double bytes) {
  const int extra = x_extra_blocks(e.n1, e.n2, e.n3h - e.kz, S * psb::xreg_threads<T, A, B>());
  constexpr size_t smem = psb::xreg_smem<T, Epi, A, B, R, S>();
  auto k = psb::xreg_kernel<T, Epi, A, B, R, S, MANY>;
  set_smem(k, smem);
  LaunchScope scope(c, what, bytes);
  launch_pdl(k, dim3((unsigned)(e.main_blocks + extra)), S * psb::xreg_threads<T, A, B>(), smem, c->stream, e, epi);
  return launch_ok(c, what);
}

template <typename T, class Epi, int A, int B, int R>
int launch_reg_x(psb_ctx* c, psb::XEpiArgs<T> e, const Epi& epi, const char* what, double bytes) {
  constexpr int C = psb::xreg_cols<T>();
  e.main_blocks = (e.kz + C - 1) / C * e.n2;
  if constexpr (x_group_wave<T, Epi, A, B, R>() > 0)
    if (e.main_blocks <= x_group_wave<T, Epi, A, B, R>()) return launch_reg_xs<T, Epi, A, B, R, 3, true>(c, e, epi, what, bytes);
  constexpr int few = psb::xreg_minb<T, Epi, A, B, R, false>();
  if constexpr (few != psb::xreg_minb<T, Epi, A, B, R, true>())
    if (e.main_blocks <= 148 * few) return launch_reg_xs<T, Epi, A, B, R, 1, false>(c, e, epi, what, bytes);
  return launch_reg_xs<T, Epi, A, B, R, 1, true>(c, e, epi, what, bytes);
}

template <typename T, class Epi, int A, int B, int R>
int launch_reg_x_batch(psb_ctx* c, const psb::XEpiArgs<T>* args, const Epi* epi, int kz, int n1, int n2, int n3h,
                       int runs, const char* what, double bytes) {
  const int extra = x_extra_blocks(n1, n2, n3h - kz, psb::xreg_threads<T, A, B>());
  constexpr int C = psb::xreg_cols<T>();
  constexpr size_t smem = psb::xreg_smem<T, Epi, A, B, R, 1>();
  const int mainb = (kz + C - 1) / C * n2;
  auto k = psb::xreg_batch<T, Epi, A, B, R>;
  set_smem(k, smem);
  LaunchScope scope(c, what, bytes);
  launch_pdl(k, dim3((unsigned)(mainb + extra), (unsigned)runs), psb::xreg_threads<T, A, B>(), smem, c->stream, args,
             epi, mainb);
  return launch_ok(c, what);
}

// f(integral constants A, B, R) for the plan of length L
template <typename T, class F>
int with_x_plan(int L, F f) {
#define PSB_CASE(LEN, A, B, R)                                                         \
  case LEN:                                                                            \
    return f(std::integral_constant<int, A>{}, std::integral_constant<int, B>{},      \
             std::integral_constant<int, R>{});
  switch (L) { PSB_REG_X(PSB_CASE) }
#undef PSB_CASE
  return PSB_ERR_SHAPE;
}

template <typename T, class Epi>
int reg_x(psb_ctx* c, const psb::XEpiArgs<T>& e, const Epi& epi, const char* what, double bytes) {
  return with_x_plan<T>(e.plan.L, [&](auto a, auto b, auto r) {
    return launch_reg_x<T, Epi, decltype(a)::value, decltype(b)::value, decltype(r)::value>(c, e, epi, what, bytes);
  });
}

template <typename T, class Epi>
int reg_x_batch(psb_ctx* c, const psb::XEpiArgs<T>* args, const Epi* epi, int L, int kz, int n1, int n2, int n3h,
                int runs, const char* what, double bytes) {
  return with_x_plan<T>(L, [&](auto a, auto b, auto r) {
    return launch_reg_x_batch<T, Epi, decltype(a)::value, decltype(b)::value, decltype(r)::value>(
        c, args, epi, kz, n1, n2, n3h, runs, what, bytes);
  });
}

#define PSB_REG_X_OF(T, ...) \
  template int reg_x<T, __VA_ARGS__>(psb_ctx*, const psb::XEpiArgs<T>&, const __VA_ARGS__&, const char*, double);
#define PSB_REG_X_BATCH_OF(T, ...)                                                                                     \
  template int reg_x_batch<T, __VA_ARGS__>(psb_ctx*, const psb::XEpiArgs<T>*, const __VA_ARGS__*, int, int, int, int, \
                                           int, int, const char*, double);

}  // namespace psbh
