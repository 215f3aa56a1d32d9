// Host side of the register z pass (psb_zreg.cuh); the psb_z_*.cu translation
// units instantiate it for one physics functor and precision each.
#pragma once
#include "psb_ctx.cuh"

namespace psbh {

// Pencils per CTA: the fewest instructions per pencil by the rounds of the three
// stages (an outer round is NT/32 * (32/B) lines, a middle round NT/A items, an
// incomplete one costs as much as a full one), against the CTAs that the shared
// memory leaves on an SM.  Five pencils where a round holds 32 lines and a job
// six fields, for instance: 30 lines each way, where four or six leave a
// quarter of the lanes idle.
template <typename T, class Phys, int A, int B>
int z_reg_best_pencils() {
  using Pl = psb::ZPlan<T, A, B>;
  using Md = psb::Mid<Phys>;
  constexpr int LW = Pl::NT / 32 * Pl::GW, QS = Pl::NT / A, MB = Pl::minb(Md::HEAVY);
  auto up = [](int a, int b) { return (a + b - 1) / b; };
  int best = 1;
  double bc = 1e30;
  for (int P = 1; P <= 32; ++P) {
    const size_t smem = psb::z_reg_smem<Phys, T, A, B>(P);
    if (smem > 200 * 1024) break;
    const int ctas = std::min<int>(MB, (int)(228 * 1024 / (smem + 1024)));
    double work = 0;
    for (int k = 0; k < Md::JOBS; ++k) {
      const int fi = Md::in0(k + 1) - Md::in0(k), fo = Md::out0(k + 1) - Md::out0(k);
      work += 30.0 * A * (up(fi * P, LW) + up(fo * P, LW));
      if (psb::phys_is_block<Phys>::value)
        work += 20.0 * B * (up(fi * P, QS) + up(fo * P, QS)) + 130.0 * up(up(P * Pl::M, 16), Pl::NT / 32);
      else
        work += 20.0 * B * (fi + fo) * up(P, QS);
    }
    // fewer resident CTAs hide less of each other's latency
    static const double hide[9] = {8, 4, 2.1, 1.25, 1.08, 1, 1, 1, 1};
    const double cost = work / P * hide[std::min(ctas, 8)];
    if (cost < bc) {
      bc = cost;
      best = P;
    }
  }
  return best;
}
// ... and two CTAs per SM over the whole launch.
template <typename T, class Phys, int A, int B>
int z_reg_pencils(long long total) {
  constexpr int NJ = psb::Mid<Phys>::JOBS;
  static const int best = z_reg_best_pencils<T, Phys, A, B>();
  int P = best;
  while (P > 1 && (total + P - 1) / P * NJ < 2 * 148) P = (P + 1) / 2;
  return P;
}

template <typename T, class Phys, int A, int B, bool P32>
int launch_reg_zp(psb_ctx* c, const psb::ZArgs<T>& z, const Phys& phys, const char* what, double bytes) {
  const int P = z_reg_pencils<T, Phys, A, B>(z.npencils);
  const size_t smem = psb::z_reg_smem<Phys, T, A, B>(P);
  auto k = psb::zreg_kernel<T, Phys, A, B, P32>;
  set_smem(k, smem);
  const long long g = persistent_grid(k, smem, (z.npencils + P - 1) / P * psb::Mid<Phys>::JOBS,
                                      psb::ZPlan<T, A, B>::NT);
  LaunchScope scope(c, what, bytes);
  const bool alone = bytes > kPdlBytes;
  c->after_z = alone ? kAfterLargeZ : kAfterNone;
  launch_pdl_if(!alone, k, dim3((unsigned)g), psb::ZPlan<T, A, B>::NT, smem, c->stream, z, phys, P);
  return launch_ok(c, what);
}

template <typename T, class Phys, int A, int B>
int launch_reg_z(psb_ctx* c, const psb::ZArgs<T>& z, const Phys& phys, const char* what, double bytes) {
  // 3/2-padded lines on both sides: k3 < M/3 stored
  if constexpr (A % 3 == 0 && (z_pad32_only<Phys>::value || std::is_same<Phys, psb::PhysProducts<T>>::value)) {
    bool pad32 = z.out_kz == 2 * A * B / 3;
    for (int f = 0; f < Phys::F_IN; ++f) pad32 = pad32 && z.in_kz[f] == 2 * A * B / 3;
    if (pad32) return launch_reg_zp<T, Phys, A, B, true>(c, z, phys, what, bytes);
    if constexpr (z_pad32_only<Phys>::value) return fail(c, PSB_ERR_SHAPE, std::string(what) + ": not 3/2-padded");
  }
  if constexpr (!z_pad32_only<Phys>::value) return launch_reg_zp<T, Phys, A, B, false>(c, z, phys, what, bytes);
  return PSB_ERR_SHAPE;
}

template <typename T, class Phys, int A, int B>
int launch_reg_z_batch(psb_ctx* c, const psb::ZArgs<T>* args, const Phys* phys, long long npencils, int runs,
                       const char* what, double bytes) {
  const int P = z_reg_pencils<T, Phys, A, B>(npencils * runs);
  const size_t smem = psb::z_reg_smem<Phys, T, A, B>(P);
  auto k = psb::zreg_batch<T, Phys, A, B>;
  set_smem(k, smem);
  const long long g = persistent_grid(k, smem, (npencils + P - 1) / P * psb::Mid<Phys>::JOBS * runs,
                                      psb::ZPlan<T, A, B>::NT);
  LaunchScope scope(c, what, bytes);
  const bool alone = bytes > kPdlBytes;
  c->after_z = alone ? kAfterLargeZ : kAfterNone;
  launch_pdl_if(!alone, k, dim3((unsigned)g), psb::ZPlan<T, A, B>::NT, smem, c->stream, args, phys, runs, P);
  return launch_ok(c, what);
}

// f(integral_constant A, integral_constant B) for the plan of M real points
template <typename T, class Phys, class F>
int with_z_plan(int M, F f, int none) {
#define PSB_CASE(H, A, B)                                                                           \
  case 2 * H:                                                                                       \
    if constexpr (z_plan_of<Phys>(H)) \
      return f(std::integral_constant<int, A>{}, std::integral_constant<int, B>{}); \
    break;
  if constexpr (sizeof(T) == 4) {
    switch (M) {
      PSB_REG_Z_F32(PSB_CASE)
      default:
        break;
    }
  } else {
    switch (M) {
      PSB_REG_Z_F64(PSB_CASE)
      default:
        break;
    }
  }
#undef PSB_CASE
  return none;
}

template <typename T, class Phys>
int reg_z(psb_ctx* c, const psb::ZArgs<T>& z, const Phys& phys, const char* what, double bytes) {
  return with_z_plan<T, Phys>(
      z.plan.L,
      [&](auto a, auto b) { return launch_reg_z<T, Phys, decltype(a)::value, decltype(b)::value>(c, z, phys, what, bytes); },
      PSB_ERR_SHAPE);
}

template <typename T, class Phys>
int reg_z_batch(psb_ctx* c, const psb::ZArgs<T>* args, const Phys* phys, int M, long long npencils, int runs,
                const char* what, double bytes) {
  return with_z_plan<T, Phys>(
      M,
      [&](auto a, auto b) {
        constexpr int A = decltype(a)::value, B = decltype(b)::value;
        if constexpr (A % 3 == 0)  // batches are 3/2-padded
          return launch_reg_z_batch<T, Phys, A, B>(c, args, phys, npencils, runs, what, bytes);
        else
          return fail(c, PSB_ERR_SHAPE, std::string(what) + ": not 3/2-padded");
      },
      PSB_ERR_SHAPE);
}

template <typename T, class Phys>
int reg_z_shape(int M, long long npencils, FFTPlan& plan) {
  return with_z_plan<T, Phys>(
      M,
      [&](auto a, auto b) {
        constexpr int A = decltype(a)::value, B = decltype(b)::value;
        plan.L = M;
        plan.npass = 3;
        for (int s = 3; s < psb::kMaxPasses; ++s) plan.radix[s] = 0;
        plan.radix[0] = A;
        plan.radix[1] = B;
        plan.radix[2] = 2;
        return z_reg_pencils<T, Phys, A, B>(npencils);
      },
      0);
}

#define PSB_REG_Z(T, ...)                                                                                     \
  template int reg_z<T, __VA_ARGS__>(psb_ctx*, const psb::ZArgs<T>&, const __VA_ARGS__&, const char*, double); \
  template int reg_z_shape<T, __VA_ARGS__>(int, long long, FFTPlan&);
#define PSB_REG_Z_BATCH(T, ...)                                                                                   \
  template int reg_z_batch<T, __VA_ARGS__>(psb_ctx*, const psb::ZArgs<T>*, const __VA_ARGS__*, int, long long, int, \
                                           const char*, double);

}  // namespace psbh
