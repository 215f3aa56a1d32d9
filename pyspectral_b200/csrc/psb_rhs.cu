// Right-hand-side pipelines of every closure and the RK4 driver.
//
// One RHS = x-inverse -> y-inverse -> fused z (c2r, products, r2c) ->
// y-forward -> x-forward fused with the spectral epilogue.  In RK mode the
// epilogue applies the stage update Q = Q0 + dt*c_i*RHS in place, so a stage
// is five kernels and the state is read twice and written once.
//
// Each of the five runs as a register pass (psb_reg.cuh, psb_zreg.cuh,
// psb_xreg.cuh) where the padded length has one, else as the staged pass of
// psb_passes.cuh with a runtime radix schedule; both give the same results to
// rounding.
#include "psb_ctx.cuh"

using namespace psb;
using namespace psbh;

namespace {

template <typename T>
KTabs<T> ktabs(const double* a, const double* b, const double* c) {
  KTabs<T> k;
  k.k1 = a;
  k.k2 = b;
  k.k3 = c;
  return k;
}

template <typename T>
AxisArgs<T> axis_common(psb_ctx* c, int L) {
  AxisArgs<T> a{};
  a.plan = *plan_for(c, L);
  a.tw = twiddles<T>(c);
  a.scale = (T)1;
  return a;
}

// ---------------------------------------------------------------------------
// 3/2-padded Navier-Stokes (DNS, Smagorinsky, SGS of filtered DNS)
// ---------------------------------------------------------------------------
// Physics that are the products (PhysProducts) of input fields 0-2 and, apart
// from them, of fields 3-5 (Phys::TWO_PRODUCTS).
template <class P, class = void>
struct two_products {
  static constexpr bool value = false;
};
template <class P>
struct two_products<P, decltype((void)P::TWO_PRODUCTS, void())> {
  static constexpr bool value = P::TWO_PRODUCTS;
};

// ts: autotuned launch shapes of the five passes (psb_autotune), or null
template <typename T, class Pre, class Phys, class Epi>
int run_ns32(psb_ctx* c, const Cx<T>* Qin, Pre pre, Phys phys, Epi epi, const psb_tuned* ts = nullptr) {
  const psb_pass_shape* sh[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  if (ts)
    for (int k = 0; k < 5; ++k) sh[k] = &ts->pass[k];
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int M1 = 3 * N1 / 2, M2 = 3 * N2 / 2, M3 = 3 * N3 / 2, Kz = N3 / 2;
  // Fi: fields after the x pass; Fb: after the y pass (the y pass's Pre may derive some)
  constexpr int Fi = Pre::F_DST, Fb = pre_b_fields<Pre>::value, Fo = Phys::F_OUT;
  static_assert(Phys::F_IN == Fb + pre_z_derived<Pre>::value, "pre/phys mismatch");
  static_assert(Epi::F_IN == Phys::F_OUT, "phys/epi mismatch");
  static_assert(pre_has_zsrc2<Pre>::value == phys_in2<Phys>::value, "means of two spectra: pre/phys mismatch");
  int st = PSB_OK;
  Cx<T>* A = scratch<T>(c, "ns.A", (size_t)Fi * M1 * N2 * Kz, &st);
  Cx<T>* B = scratch<T>(c, "ns.B", (size_t)Fb * M1 * M2 * Kz, &st);
  Cx<T>* C = scratch<T>(c, "ns.C", (size_t)Fo * M1 * M2 * Kz, &st);
  Cx<T>* D = scratch<T>(c, "ns.D", (size_t)Fo * M1 * N2 * Kz, &st);
  if (st != PSB_OK) return st;
  if (!Qin) return PSB_OK;  // allocation only
  const long long fsN = (long long)N1 * N2 * N3h;
  // x inverse: spectral rows k1 -> padded positions
  AxisArgs<T> a = axis_common<T>(c, M1);
  a.in = Qin;
  a.out = A;
  a.in_fstride = fsN;
  a.in_ostride = N3h;
  a.in_rstride = (long long)N2 * N3h;
  a.out_fstride = (long long)M1 * N2 * Kz;
  a.out_ostride = Kz;
  a.out_rstride = (long long)N2 * Kz;
  a.nouter = N2;
  a.ncols = Kz;
  a.in_rows = N1;
  a.out_rows = M1;
  a.in_map = map_pad32(N1);
  a.out_map = map_id(M1);
  a.k_row = c->kx;
  a.k_outer = c->ky;
  a.k_col = c->kz;
  PSB_TRY((launch_axis<T, true, Pre, true>(c, a, pre, "x-inverse", sh[0])));
  // y inverse (fields folded into the outer index)
  AxisArgs<T> b = axis_common<T>(c, M2);
  b.in = A;
  b.out = B;
  b.in_ostride = (long long)N2 * Kz;
  b.in_rstride = Kz;
  b.out_ostride = (long long)M2 * Kz;
  b.out_rstride = Kz;
  using YP = pre_ypass<T, Pre>;
  b.nouter = YP::groups * M1;
  b.in_fstride = (long long)YP::in_fields * M1 * N2 * Kz;
  b.out_fstride = (long long)YP::out_fields * M1 * M2 * Kz;
  b.ncols = Kz;
  b.in_rows = N2;
  b.out_rows = M2;
  b.in_map = map_pad32(N2);
  b.out_map = map_id(M2);
  b.k_row = c->ky;
  const double s32 = std::sqrt(std::pow(1.5, 3) * std::sqrt((double)N1 * N2 * N3));
  const double fac = s32 / ((double)M1 * M2 * M3), fsc = field_scale(fac);
  b.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true, typename YP::type, true>(c, b, typename YP::type{}, "y-inverse", sh[1])));
  // fused z
  ZArgs<T> z{};
  const long long fsP = (long long)M1 * M2 * Kz;
  set_z_inputs<T, Pre, Phys::F_IN>(z, B, fsP, Kz, c->kz);
  for (int g = 0; g < Fo; ++g) {
    z.out[g] = C + g * fsP;
    z.out_pstride[g] = Kz;
  }
  z.out_kz = Kz;
  z.npencils = (long long)M1 * M2;
  z.fac = (T)(fac / fsc);
  z.plan = *plan_for(c, M3);
  z.tw = twiddles<T>(c);
  // two products passes in the registers against one staged pass of both sets
  // (64^3 FP64 42 us against 133); where the length has no register pass the one
  // staged launch is the faster (12^3, 18 points, FP64 16.7 us against 29.6)
  bool split = false;
  if constexpr (two_products<Phys>::value) {
    split = c->use_zrr && has_reg_z<T, PhysProducts<T>>(M3);
    for (int h = 0; split && h < 2; ++h) {
      ZArgs<T> y = z;
      for (int f = 0; f < 3; ++f) {
        y.in[f] = z.in[3 * h + f];
        y.in_pstride[f] = z.in_pstride[3 * h + f];
        y.in_kz[f] = z.in_kz[3 * h + f];
      }
      for (int g = 0; g < 6; ++g) {
        y.out[g] = z.out[6 * h + g];
        y.out_pstride[g] = z.out_pstride[6 * h + g];
      }
      PSB_TRY((launch_z<T, PhysProducts<T>, true>(c, y, PhysProducts<T>{}, "z-fused")));
    }
  }
  if (!split) PSB_TRY((launch_z<T, Phys, true>(c, z, phys, "z-fused", 0.0, sh[2])));
  // y forward with truncation
  AxisArgs<T> d = axis_common<T>(c, M2);
  d.in = C;
  d.out = D;
  d.in_ostride = (long long)M2 * Kz;
  d.in_rstride = Kz;
  d.out_ostride = (long long)N2 * Kz;
  d.out_rstride = Kz;
  d.nouter = Fo * M1;
  d.ncols = Kz;
  d.in_rows = M2;
  d.out_rows = N2;
  d.in_map = map_id(M2);
  d.out_map = map_pad32(N2);
  PSB_TRY((launch_axis<T, false, PreCopy<T>, true>(c, d, PreCopy<T>{}, "y-forward", sh[3])));
  // x forward + epilogue
  XEpiArgs<T> e{};
  e.in = D;
  e.in_fstride = (long long)M1 * N2 * Kz;
  e.in_rstride = (long long)N2 * Kz;
  e.in_ostride = Kz;
  e.n1 = N1;
  e.n2 = N2;
  e.n3h = N3h;
  e.kz = Kz;
  e.out_map = map_pad32(N1);
  e.plan = *plan_for(c, M1);
  e.tw = twiddles<T>(c);
  return launch_epi<T, Epi, true>(c, e, epi, "x-forward+epilogue", sh[4]);
}

// Products of u and of the sharp-cutoff filtered u for computeSGS_DNS
// (PySpectral/src/Classes.py:861-915)
template <typename T>
struct PreFiltered {
  static constexpr int F_SRC = 3, F_DST = 6;
  const double *g1, *g2, *g3;
  __device__ void operator()(int i, int o, int cc, const AxisArgs<T>&, const Cx<T>* s, Cx<T>* d) const {
    const T g = (T)(g1[i] * g2[o] * g3[cc]);
    d[0] = s[0];
    d[1] = s[1];
    d[2] = s[2];
    d[3] = g * s[0];
    d[4] = g * s[1];
    d[5] = g * s[2];
  }
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t = copy_fields<T>(6, g1, g2, g3);
    for (int f = 3; f < 6; ++f) t.sa[f] = (unsigned char)(f - 3);
    t.mfrom = 3;
    return t;
  }
};

// test filter applied on load (PySpectral/src/Classes.py:147-150)
template <typename T>
struct PreMask3 {
  static constexpr int F_SRC = 3, F_DST = 3;
  const double *g1, *g2, *g3;
  __device__ void operator()(int i, int o, int cc, const AxisArgs<T>&, const Cx<T>* s, Cx<T>* d) const {
    const T g = (T)(g1[i] * g2[o] * g3[cc]);
    d[0] = g * s[0];
    d[1] = g * s[1];
    d[2] = g * s[2];
  }
  __host__ FieldTab<T> fields() const { return copy_fields<T>(3, g1, g2, g3); }
};

template <typename T>
struct PhysSGSDNS {
  static constexpr int F_IN = 6, F_OUT = 12;
  static constexpr bool TWO_PRODUCTS = true;
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const T u = in[3 * h], v = in[3 * h + 1], w = in[3 * h + 2];
      out[6 * h + 0] = u * u;
      out[6 * h + 1] = v * v;
      out[6 * h + 2] = w * w;
      out[6 * h + 3] = u * v;
      out[6 * h + 4] = u * w;
      out[6 * h + 5] = v * w;
    }
  }
};

// tau_ij = Gf*(u_i u_j)^ - (Gf u_i Gf u_j)^ and its projected divergence
// (PySpectral/src/Classes.py:917-928)
template <typename T>
struct EpiSGSDNS {
  static constexpr int F_IN = 12;
  __host__ double io_bytes(long long npts) const {
    return (double)sizeof(Cx<T>) * npts * (3 + (tau ? 6 : 0));
  }
  KTabs<T> k;
  const double *g1, *g2, *g3;
  Cx<T>* w0;
  Cx<T>* tau;
  long long fstride;
  int n2, n3h;
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const {
    const long long s = ((long long)i1 * n2 + i2) * n3h + i3;
    const T g = (T)(g1[i1] * g2[i2] * g3[i3]);
    Cx<T> t[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) t[m] = g * P[m] - P[6 + m];
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    const Cx<T> kk = (k1 * k1) * t[0] + (k2 * k2) * t[1] + (k3 * k3) * t[2] + ((T)2 * k1 * k2) * t[3] +
                     ((T)2 * k1 * k3) * t[4] + ((T)2 * k2 * k3) * t[5];
    const Cx<T> proj = mul_i(ksqi * kk);
    w0[s] = mik(k1, t[0]) + mik(k2, t[3]) + mik(k3, t[4]) + pik(k1, proj);
    w0[fstride + s] = mik(k1, t[3]) + mik(k2, t[1]) + mik(k3, t[5]) + pik(k2, proj);
    w0[2 * fstride + s] = mik(k1, t[4]) + mik(k2, t[5]) + mik(k3, t[2]) + pik(k3, proj);
    if (tau) {
#pragma unroll
      for (int m = 0; m < 6; ++m) tau[m * fstride + s] = t[m];
    }
  }
};

// ---------------------------------------------------------------------------
// MHD: unpadded transforms under the 2/3 rule
// ---------------------------------------------------------------------------
template <typename T, class Pre, class Phys, class Epi>
int run_n23(psb_ctx* c, const Cx<T>* Qin, Pre pre, Phys phys, Epi epi) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int Kz = c->kz_mhd;
  constexpr int Fi = Phys::F_IN, Fo = Phys::F_OUT;
  static_assert(Pre::F_DST == Fi && Epi::F_IN == Fo, "pass field counts");
  int st = PSB_OK;
  Cx<T>* A = scratch<T>(c, "mhd.A", (size_t)Fi * N1 * N2 * Kz, &st);
  Cx<T>* B = scratch<T>(c, "mhd.B", (size_t)Fi * N1 * N2 * Kz, &st);
  Cx<T>* C = scratch<T>(c, "mhd.C", (size_t)Fo * N1 * N2 * Kz, &st);
  Cx<T>* D = scratch<T>(c, "mhd.D", (size_t)Fo * N1 * N2 * Kz, &st);
  if (st != PSB_OK) return st;
  if (!Qin) return PSB_OK;
  const long long fsN = (long long)N1 * N2 * N3h;
  const long long fsP = (long long)N1 * N2 * Kz;
  AxisArgs<T> a = axis_common<T>(c, N1);
  a.in = Qin;
  a.out = A;
  a.in_fstride = fsN;
  a.in_ostride = N3h;
  a.in_rstride = (long long)N2 * N3h;
  a.out_fstride = fsP;
  a.out_ostride = Kz;
  a.out_rstride = (long long)N2 * Kz;
  a.nouter = N2;
  a.ncols = Kz;
  a.in_rows = N1;
  a.out_rows = N1;
  a.in_map = map_id(N1);
  a.out_map = map_id(N1);
  PSB_TRY((launch_axis<T, true>(c, a, pre, "mhd x-inverse")));
  AxisArgs<T> b = axis_common<T>(c, N2);
  b.in = A;
  b.out = B;
  b.in_ostride = (long long)N2 * Kz;
  b.in_rstride = Kz;
  b.out_ostride = (long long)N2 * Kz;
  b.out_rstride = Kz;
  b.nouter = Fi * N1;
  b.ncols = Kz;
  b.in_rows = N2;
  b.out_rows = N2;
  b.in_map = map_id(N2);
  b.out_map = map_id(N2);
  const double fac = 1.0 / ((double)N1 * N2 * N3), fsc = field_scale(fac);
  b.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true>(c, b, PreCopy<T>{}, "mhd y-inverse")));
  ZArgs<T> z{};
  for (int f = 0; f < Fi; ++f) {
    z.in[f] = B + f * fsP;
    z.in_pstride[f] = Kz;
    z.in_kz[f] = Kz;
  }
  for (int g = 0; g < Fo; ++g) {
    z.out[g] = C + g * fsP;
    z.out_pstride[g] = Kz;
  }
  z.out_kz = Kz;
  z.npencils = (long long)N1 * N2;
  z.fac = (T)(fac / fsc);
  z.plan = *plan_for(c, N3);
  z.tw = twiddles<T>(c);
  PSB_TRY(launch_z<T>(c, z, phys, "mhd z-fused"));
  AxisArgs<T> d = axis_common<T>(c, N2);
  d.in = C;
  d.out = D;
  d.in_ostride = (long long)N2 * Kz;
  d.in_rstride = Kz;
  d.out_ostride = (long long)N2 * Kz;
  d.out_rstride = Kz;
  d.nouter = Fo * N1;
  d.ncols = Kz;
  d.in_rows = N2;
  d.out_rows = N2;
  d.in_map = map_id(N2);
  d.out_map = map_id(N2);
  PSB_TRY((launch_axis<T, false>(c, d, PreCopy<T>{}, "mhd y-forward")));
  XEpiArgs<T> e{};
  e.in = D;
  e.in_fstride = fsP;
  e.in_rstride = (long long)N2 * Kz;
  e.in_ostride = Kz;
  e.n1 = N1;
  e.n2 = N2;
  e.n3h = N3h;
  e.kz = Kz;
  e.out_map = map_id(N1);
  e.plan = *plan_for(c, N1);
  e.tw = twiddles<T>(c);
  return launch_epi<T>(c, e, epi, "mhd x-forward+epilogue");
}

// MHD of the MPI solver: the 2/3-masked fields (u, B) -> (u_iu_j - B_iB_j, u x B)
template <typename T>
int run_mhd(psb_ctx* c, const Cx<T>* Qin, EpiMHD<T> epi) {
  return run_n23<T>(c, Qin, PreMask6<T>{c->mx, c->my, c->mz}, PhysMHD<T>{}, epi);
}

// ---------------------------------------------------------------------------
// 2x-padded memory closures (t-model, static and dynamic tau-model)
// ---------------------------------------------------------------------------
struct MemCfg {
  const char* tag;     // scratch name prefix
  const double* filt;  // test filter masks (N grid) or null
  int kfp;             // test-filter split (0 = seperateModes)
  bool want_plp;
  bool want_box;
  int kfb;
};

// Stage A: u -> PL on the full 2x grid (q part and unpad_2x part).
template <typename T>
int run_pl(psb_ctx* c, const Cx<T>* Qin, const psb_params* p, const MemCfg& m, Cx<T>** B2_out,
           Cx<T>** PLq_out, Cx<T>* PLp, Cx<T>* Lbox, Cx<T>* PLfull = nullptr) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int F1 = 2 * N1, F2 = 2 * N2, F3 = 2 * N3, F3h = N3 + 1, Kz = N3 / 2;
  int st = PSB_OK;
  std::string t = m.tag;
  Cx<T>* A2 = scratch<T>(c, (t + ".A2").c_str(), (size_t)3 * F1 * N2 * Kz, &st);
  Cx<T>* B2 = scratch<T>(c, (t + ".B2").c_str(), (size_t)3 * F1 * F2 * Kz, &st);
  Cx<T>* C2 = scratch<T>(c, "mem.C2", (size_t)6 * F1 * F2 * F3h, &st);
  Cx<T>* D2 = scratch<T>(c, "mem.D2", (size_t)6 * F1 * F2 * F3h, &st);
  Cx<T>* E = scratch<T>(c, (t + ".E").c_str(), (size_t)3 * F1 * F2 * F3h, &st);
  if (st != PSB_OK) return st;
  *B2_out = B2;
  *PLq_out = E;
  if (!Qin) return PSB_OK;
  const long long fsN = (long long)N1 * N2 * N3h;
  AxisArgs<T> a = axis_common<T>(c, F1);
  a.in = Qin;
  a.out = A2;
  a.in_fstride = fsN;
  a.in_ostride = N3h;
  a.in_rstride = (long long)N2 * N3h;
  a.out_fstride = (long long)F1 * N2 * Kz;
  a.out_ostride = Kz;
  a.out_rstride = (long long)N2 * Kz;
  a.nouter = N2;
  a.ncols = Kz;
  a.in_rows = N1;
  a.out_rows = F1;
  a.in_map = map_pad2x_nyq0(N1);
  a.out_map = map_id(F1);
  a.k_row = c->kx;
  a.k_outer = c->ky;
  a.k_col = c->kz;
  if (m.filt) {
    PSB_TRY((launch_axis<T, true>(c, a, PreMask3<T>{m.filt, m.filt + N1, m.filt + N1 + N2},
                                  "2x x-inverse (test-filtered)")));
  } else {
    PSB_TRY((launch_axis<T, true>(c, a, PreCopyN<T, 3>{}, "2x x-inverse")));
  }
  AxisArgs<T> b = axis_common<T>(c, F2);
  b.in = A2;
  b.out = B2;
  b.in_ostride = (long long)N2 * Kz;
  b.in_rstride = Kz;
  b.out_ostride = (long long)F2 * Kz;
  b.out_rstride = Kz;
  b.nouter = 3 * F1;
  b.ncols = Kz;
  b.in_rows = N2;
  b.out_rows = F2;
  b.in_map = map_pad2x_nyq0(N2);
  b.out_map = map_id(F2);
  const double s2 = std::sqrt(8.0 * std::sqrt((double)N1 * N2 * N3));
  const double fac = s2 / ((double)F1 * F2 * F3), fsc = field_scale(fac);
  b.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true>(c, b, PreCopy<T>{}, "2x y-inverse")));
  ZArgs<T> z{};
  const long long fsB = (long long)F1 * F2 * Kz, fsC = (long long)F1 * F2 * F3h;
  for (int f = 0; f < 3; ++f) {
    z.in[f] = B2 + f * fsB;
    z.in_pstride[f] = Kz;
    z.in_kz[f] = Kz;
  }
  for (int g = 0; g < 6; ++g) {
    z.out[g] = C2 + g * fsC;
    z.out_pstride[g] = F3h;
  }
  z.out_kz = F3h;
  z.npencils = (long long)F1 * F2;
  z.fac = (T)(fac / fsc);
  z.plan = *plan_for(c, F3);
  z.tw = twiddles<T>(c);
  PSB_TRY(launch_z<T>(c, z, PhysProducts<T>{}, "2x z-products"));
  AxisArgs<T> d = axis_common<T>(c, F2);
  d.in = C2;
  d.out = D2;
  d.in_ostride = (long long)F2 * F3h;
  d.in_rstride = F3h;
  d.out_ostride = (long long)F2 * F3h;
  d.out_rstride = F3h;
  d.nouter = 6 * F1;
  d.ncols = F3h;
  d.in_rows = F2;
  d.out_rows = F2;
  d.in_map = map_id(F2);
  d.out_map = map_id(F2);
  PSB_TRY((launch_axis<T, false>(c, d, PreCopy<T>{}, "2x y-forward")));
  EpiPL<T> epi{};
  epi.Q = Qin;
  epi.fstride_n = fsN;
  epi.N1 = N1;
  epi.N2 = N2;
  epi.N3 = N3;
  epi.n3h = N3h;
  epi.nf2 = F2;
  epi.nf3h = F3h;
  epi.fstride_2x = fsC;
  epi.kf = ktabs<T>(c->kxf, c->kyf, c->kzf);
  epi.nu = (T)p->nu;
  epi.rotate = p->rotate;
  epi.Om1 = (T)p->Om1;
  epi.Om2 = (T)p->Om2;
  epi.Om3 = (T)p->Om3;
  epi.filt = m.filt;
  epi.kfp = m.kfp;
  epi.PLq = E;
  epi.PLp = PLp;
  epi.Lbox = Lbox;
  epi.kfb = m.kfb;
  epi.PLfull = PLfull;
  XEpiArgs<T> e{};
  e.in = D2;
  e.in_fstride = fsC;
  e.in_rstride = (long long)F2 * F3h;
  e.in_ostride = F3h;
  e.n1 = F1;
  e.n2 = F2;
  e.n3h = F3h;
  e.kz = F3h;
  e.out_map = map_id(F1);
  e.plan = *plan_for(c, F1);
  e.tw = twiddles<T>(c);
  return launch_epi<T>(c, e, epi, "2x x-forward+PL");
}

// Stage B: PLQL from u (B2) and PL_q (E) -> products -> N-grid epilogue.
// FULL: the products stay on the whole 2x grid (every k3 of the 2x grid, 2N2
// rows, 2N1 rows) and the epilogue runs there (EpiPLQLFull); otherwise they
// are truncated to the N grid (unpad_2x) on the way out.  An epilogue of six
// spectra gets the symmetric products (EpiPLQL), one of nine every product
// (EpiStore<T, 9>, EpiPLQLFull).
template <typename T, class Epi = EpiPLQL<T>, bool FULL = false>
int run_plql(psb_ctx* c, const MemCfg& m, Cx<T>* B2, Cx<T>* E, Epi epi) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int F1 = 2 * N1, F2 = 2 * N2, F3 = 2 * N3, F3h = N3 + 1, Kz = N3 / 2;
  // output k3 count and y rows of the forward passes
  const int KO = FULL ? F3h : Kz, RY = FULL ? F2 : N2;
  int st = PSB_OK;
  Cx<T>* A3 = scratch<T>(c, "mem.A3", (size_t)3 * F1 * F2 * F3h, &st);
  Cx<T>* B3 = scratch<T>(c, "mem.B3", (size_t)3 * F1 * F2 * F3h, &st);
  // nine products u_j q_i, or the six symmetric sums of them
  using Phys = std::conditional_t<Epi::F_IN == 6, PhysPLQS<T>, PhysPLQL<T>>;
  constexpr int FO = Phys::F_OUT;
  static_assert(Epi::F_IN == FO, "phys/epi mismatch");
  Cx<T>* C3 = scratch<T>(c, FULL ? "mem.C3f" : (FO == 6 ? "mem.C3s" : "mem.C3"), (size_t)FO * F1 * F2 * KO, &st);
  Cx<T>* D3 = scratch<T>(c, FULL ? "mem.D3f" : (FO == 6 ? "mem.D3s" : "mem.D3"), (size_t)FO * F1 * RY * KO, &st);
  if (st != PSB_OK) return st;
  if (!B2) return PSB_OK;
  const long long fsC = (long long)F1 * F2 * F3h;
  AxisArgs<T> a = axis_common<T>(c, F1);
  a.in = E;
  a.out = A3;
  a.in_fstride = fsC;
  a.in_ostride = F3h;
  a.in_rstride = (long long)F2 * F3h;
  a.out_fstride = fsC;
  a.out_ostride = F3h;
  a.out_rstride = (long long)F2 * F3h;
  a.nouter = F2;
  a.ncols = F3h;
  a.in_rows = F1;
  a.out_rows = F1;
  a.in_map = map_id(F1);
  a.out_map = map_id(F1);
  PSB_TRY((launch_axis<T, true>(c, a, PreCopyN<T, 3>{}, "PLq x-inverse")));
  AxisArgs<T> b = axis_common<T>(c, F2);
  b.in = A3;
  b.out = B3;
  b.in_ostride = (long long)F2 * F3h;
  b.in_rstride = F3h;
  b.out_ostride = (long long)F2 * F3h;
  b.out_rstride = F3h;
  b.nouter = 3 * F1;
  b.ncols = F3h;
  b.in_rows = F2;
  b.out_rows = F2;
  b.in_map = map_id(F2);
  b.out_map = map_id(F2);
  // u in B2 carries the same power of two (run_pl)
  const double s2 = std::sqrt(8.0 * std::sqrt((double)N1 * N2 * N3));
  const double fac = s2 / ((double)F1 * F2 * F3), fsc = field_scale(fac);
  b.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true>(c, b, PreCopy<T>{}, "PLq y-inverse")));
  ZArgs<T> z{};
  const long long fsB = (long long)F1 * F2 * Kz;
  for (int f = 0; f < 3; ++f) {
    z.in[f] = B2 + f * fsB;
    z.in_pstride[f] = Kz;
    z.in_kz[f] = Kz;
    z.in[3 + f] = B3 + f * fsC;
    z.in_pstride[3 + f] = F3h;
    z.in_kz[3 + f] = F3h;
  }
  const long long fsO = (long long)F1 * F2 * KO;
  for (int g = 0; g < FO; ++g) {
    z.out[g] = C3 + g * fsO;
    z.out_pstride[g] = KO;
  }
  z.out_kz = KO;
  z.npencils = (long long)F1 * F2;
  z.fac = (T)(fac / fsc);
  z.plan = *plan_for(c, F3);
  z.tw = twiddles<T>(c);
  PSB_TRY(launch_z<T>(c, z, Phys{}, "PLQL z-products"));
  AxisArgs<T> d = axis_common<T>(c, F2);
  d.in = C3;
  d.out = D3;
  d.in_ostride = (long long)F2 * KO;
  d.in_rstride = KO;
  d.out_ostride = (long long)RY * KO;
  d.out_rstride = KO;
  d.nouter = FO * F1;
  d.ncols = KO;
  d.in_rows = F2;
  d.out_rows = RY;
  d.in_map = map_id(F2);
  d.out_map = FULL ? map_id(F2) : map_pad2x(N2);
  PSB_TRY((launch_axis<T, false>(c, d, PreCopy<T>{}, "PLQL y-forward")));
  XEpiArgs<T> e{};
  e.in = D3;
  e.in_fstride = (long long)F1 * RY * KO;
  e.in_rstride = (long long)RY * KO;
  e.in_ostride = KO;
  e.n1 = FULL ? F1 : N1;
  e.n2 = RY;
  e.n3h = FULL ? F3h : N3h;
  e.kz = KO;
  e.out_map = FULL ? map_id(F1) : map_pad2x(N1);
  e.plan = *plan_for(c, F1);
  e.tw = twiddles<T>(c);
  return launch_epi<T>(c, e, epi, "PLQL x-forward+epilogue");
}

// ---------------------------------------------------------------------------
// MHD t-model: plain MHD RHS (2/3 rule, N grid) + Ct t PLQL from two 2x-grid
// stages.  Stage A: (u, B) -> nine products -> QL on the 2x grid.  Stage B:
// (u, B) and QL -> nine linearised products -> PLQL on the N grid, fused with
// the RK stage update.
// ---------------------------------------------------------------------------
template <typename T>
int run_mhd_tmodel(psb_ctx* c, StepIO<T> io, const psb_params* p) {
  const Cx<T>* Qin = io.Q;
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int F1 = 2 * N1, F2 = 2 * N2, F3 = 2 * N3, F3h = N3 + 1, Kz = c->kz_mhd;
  const long long fsN = (long long)N1 * N2 * N3h, fsC = (long long)F1 * F2 * F3h;
  int st = PSB_OK;
  Cx<T>* R6 = scratch<T>(c, "mt.R6", (size_t)6 * fsN, &st);
  Cx<T>* A2 = scratch<T>(c, "mt.A2", (size_t)6 * F1 * N2 * Kz, &st);
  Cx<T>* B2 = scratch<T>(c, "mt.B2", (size_t)6 * F1 * F2 * Kz, &st);
  Cx<T>* C2 = scratch<T>(c, "mt.C2", (size_t)9 * fsC, &st);  // products; later QL x-inverse, PLQL y-forward
  Cx<T>* D2 = scratch<T>(c, "mt.D2", (size_t)9 * fsC, &st);  // products y-forward; later QL y-inverse
  Cx<T>* E = scratch<T>(c, "mt.E", (size_t)6 * fsC, &st);    // QL; later the linearised products
  if (st != PSB_OK) return st;
  const double* m1 = c->mx;
  const double* m2 = c->my;
  const double* m3 = c->mz;
  const T nu = (T)p->nu, eta = (T)(p->eta < 0 ? p->nu : p->eta);
  StepIO<T> ior = io;
  ior.mode = kRHS;
  ior.rhs_out = R6;
  ior.comp = nullptr;
  ior.w0_out = nullptr;
  EpiMHD<T> plain{ior, ktabs<T>(c->kx, c->ky, c->kz), m1, m2, m3, reinterpret_cast<const Cx<T>*>(p->force), nu,
                  eta};
  PSB_TRY(run_mhd<T>(c, Qin, plain));
  if (!Qin) return PSB_OK;
  const double fac = 1.0 / ((double)N1 * N2 * N3), fsc = field_scale(fac);
  const double down = (double)N1 * N2 * N3 / ((double)F1 * F2 * F3);
  // stage A: masked (u, B) onto the 2x grid
  AxisArgs<T> a = axis_common<T>(c, F1);
  a.in = Qin;
  a.out = A2;
  a.in_fstride = fsN;
  a.in_ostride = N3h;
  a.in_rstride = (long long)N2 * N3h;
  a.out_fstride = (long long)F1 * N2 * Kz;
  a.out_ostride = Kz;
  a.out_rstride = (long long)N2 * Kz;
  a.nouter = N2;
  a.ncols = Kz;
  a.in_rows = N1;
  a.out_rows = F1;
  a.in_map = map_pad2x(N1);
  a.out_map = map_id(F1);
  PSB_TRY((launch_axis<T, true>(c, a, PreMask6<T>{m1, m2, m3}, "mhd-t 2x x-inverse")));
  AxisArgs<T> b = axis_common<T>(c, F2);
  b.in = A2;
  b.out = B2;
  b.in_ostride = (long long)N2 * Kz;
  b.in_rstride = Kz;
  b.out_ostride = (long long)F2 * Kz;
  b.out_rstride = Kz;
  b.nouter = 6 * F1;
  b.ncols = Kz;
  b.in_rows = N2;
  b.out_rows = F2;
  b.in_map = map_pad2x(N2);
  b.out_map = map_id(F2);
  b.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true>(c, b, PreCopy<T>{}, "mhd-t 2x y-inverse")));
  ZArgs<T> z{};
  const long long fsB = (long long)F1 * F2 * Kz;
  for (int f = 0; f < 6; ++f) {
    z.in[f] = B2 + f * fsB;
    z.in_pstride[f] = Kz;
    z.in_kz[f] = Kz;
  }
  for (int g = 0; g < 9; ++g) {
    z.out[g] = C2 + g * fsC;
    z.out_pstride[g] = F3h;
  }
  z.out_kz = F3h;
  z.npencils = (long long)F1 * F2;
  z.fac = (T)(fac / fsc);
  z.plan = *plan_for(c, F3);
  z.tw = twiddles<T>(c);
  PSB_TRY(launch_z<T>(c, z, PhysMHD<T>{}, "mhd-t 2x z-products"));
  AxisArgs<T> d = axis_common<T>(c, F2);
  d.in = C2;
  d.out = D2;
  d.in_ostride = (long long)F2 * F3h;
  d.in_rstride = F3h;
  d.out_ostride = (long long)F2 * F3h;
  d.out_rstride = F3h;
  d.nouter = 9 * F1;
  d.ncols = F3h;
  d.in_rows = F2;
  d.out_rows = F2;
  d.in_map = map_id(F2);
  d.out_map = map_id(F2);
  PSB_TRY((launch_axis<T, false>(c, d, PreCopy<T>{}, "mhd-t 2x y-forward")));
  EpiMHDQ<T> eq{ktabs<T>(c->kxf, c->kyf, c->kzf), m1, m2, m3, N1, N2, N3h, F2, F3h, fsC, (T)down, E};
  XEpiArgs<T> e{};
  e.in = D2;
  e.in_fstride = fsC;
  e.in_rstride = (long long)F2 * F3h;
  e.in_ostride = F3h;
  e.n1 = F1;
  e.n2 = F2;
  e.n3h = F3h;
  e.kz = F3h;
  e.out_map = map_id(F1);
  e.plan = *plan_for(c, F1);
  e.tw = twiddles<T>(c);
  PSB_TRY(launch_epi<T>(c, e, eq, "mhd-t 2x x-forward+QL"));
  // stage B: QL back to physical space next to (u, B)
  Cx<T>* A3 = C2;
  Cx<T>* B3 = D2;
  AxisArgs<T> a3 = axis_common<T>(c, F1);
  a3.in = E;
  a3.out = A3;
  a3.in_fstride = fsC;
  a3.in_ostride = F3h;
  a3.in_rstride = (long long)F2 * F3h;
  a3.out_fstride = fsC;
  a3.out_ostride = F3h;
  a3.out_rstride = (long long)F2 * F3h;
  a3.nouter = F2;
  a3.ncols = F3h;
  a3.in_rows = F1;
  a3.out_rows = F1;
  a3.in_map = map_id(F1);
  a3.out_map = map_id(F1);
  PSB_TRY((launch_axis<T, true>(c, a3, PreCopyN<T, 6>{}, "mhd-t QL x-inverse")));
  AxisArgs<T> b3 = axis_common<T>(c, F2);
  b3.in = A3;
  b3.out = B3;
  b3.in_ostride = (long long)F2 * F3h;
  b3.in_rstride = F3h;
  b3.out_ostride = (long long)F2 * F3h;
  b3.out_rstride = F3h;
  b3.nouter = 6 * F1;
  b3.ncols = F3h;
  b3.in_rows = F2;
  b3.out_rows = F2;
  b3.in_map = map_id(F2);
  b3.out_map = map_id(F2);
  b3.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true>(c, b3, PreCopy<T>{}, "mhd-t QL y-inverse")));
  Cx<T>* C3 = E;
  Cx<T>* D3 = C2;
  ZArgs<T> z3{};
  for (int f = 0; f < 6; ++f) {
    z3.in[f] = B2 + f * fsB;
    z3.in_pstride[f] = Kz;
    z3.in_kz[f] = Kz;
    z3.in[6 + f] = B3 + f * fsC;
    z3.in_pstride[6 + f] = F3h;
    z3.in_kz[6 + f] = F3h;
  }
  for (int g = 0; g < 9; ++g) {
    z3.out[g] = C3 + g * fsB;
    z3.out_pstride[g] = Kz;
  }
  z3.out_kz = Kz;
  z3.npencils = (long long)F1 * F2;
  z3.fac = (T)(fac / fsc);
  z3.plan = *plan_for(c, F3);
  z3.tw = twiddles<T>(c);
  PSB_TRY(launch_z<T>(c, z3, PhysMHDLin<T>{}, "mhd-t PLQL z-products"));
  AxisArgs<T> d3 = axis_common<T>(c, F2);
  d3.in = C3;
  d3.out = D3;
  d3.in_ostride = (long long)F2 * Kz;
  d3.in_rstride = Kz;
  d3.out_ostride = (long long)N2 * Kz;
  d3.out_rstride = Kz;
  d3.nouter = 9 * F1;
  d3.ncols = Kz;
  d3.in_rows = F2;
  d3.out_rows = N2;
  d3.in_map = map_id(F2);
  d3.out_map = map_pad2x(N2);
  PSB_TRY((launch_axis<T, false>(c, d3, PreCopy<T>{}, "mhd-t PLQL y-forward")));
  EpiMHDT<T> et{io, ktabs<T>(c->kx, c->ky, c->kz), m1, m2, m3, R6, (T)(p->Ct * p->t * down), io.w0_out};
  XEpiArgs<T> e3{};
  e3.in = D3;
  e3.in_fstride = (long long)F1 * N2 * Kz;
  e3.in_rstride = (long long)N2 * Kz;
  e3.in_ostride = Kz;
  e3.n1 = N1;
  e3.n2 = N2;
  e3.n3h = N3h;
  e3.kz = Kz;
  e3.out_map = map_pad2x(N1);
  e3.plan = *plan_for(c, F1);
  e3.tw = twiddles<T>(c);
  return launch_epi<T>(c, e3, et, "mhd-t PLQL x-forward+epilogue");
}

// ---------------------------------------------------------------------------
// Dynamic Smagorinsky (PySpectral/src/RHSfunctions.py:1663-1862)
//
// Two pipeline passes store, for u and for the test-filtered u~, the six
// dealiased products and the six |S| S_ij spectra (PhysSmag with
// (Cs Delta)^2 = -1/2 gives |S| S_ij exactly).  One FP64 reduction forms
// L = F(uu) - (u~u~), M = -2 Delta^2 (alpha^2 |S~|S~ - F(|S|S)) point by point
// and Cs^2 = <L:M>/<M:M>; the reference takes both means on the 3/2 grid
// after pad(), which by Parseval is the spectral sum over the modes pad()
// keeps (k3 > 0 twice; the k3 = 0 plane as c2r reads it, i.e. its Hermitian
// part).  The Smagorinsky epilogue then runs on the stored u spectra with
// tau = -2 Cs^2 Delta^2 (|S| S)^ read from the device: no host round trip.
// ---------------------------------------------------------------------------
// myFilter(uhat, kL) (src/Classes.py:1271-1279) on load, then the strain of PreStrain
template <typename T>
struct PreStrainFiltered : PreStrain<T> {
  const double *g1, *g2, *g3;
  PreStrainFiltered(const double* a, const double* b, const double* c) : g1(a), g2(b), g3(c) {}
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t = PreStrain<T>::fields();
    t.m1 = g1;
    t.m2 = g2;
    t.m3 = g3;
    return t;
  }
  __device__ void operator()(int i, int o, int cc, const AxisArgs<T>& a, const Cx<T>* s, Cx<T>* d) const {
    const T g = (T)(g1[i] * g2[o] * g3[cc]);
    const Cx<T> f[3] = {g * s[0], g * s[1], g * s[2]};
    PreStrain<T>::operator()(i, o, cc, a, f, d);
  }
};

constexpr int kLmBlocks = 296;

template <typename T>
__device__ __forceinline__ void dsmag_lm(const Cx<T>* __restrict__ A, const Cx<T>* __restrict__ B, long long fs,
                                         long long s, double g, double d2, double* Lr, double* Li, double* Mr,
                                         double* Mi) {
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const Cx<T> a = A[m * fs + s], b = B[m * fs + s];
    const Cx<T> sa = A[(6 + m) * fs + s], sb = B[(6 + m) * fs + s];
    Lr[m] = g * (double)a.x - (double)b.x;
    Li[m] = g * (double)a.y - (double)b.y;
    Mr[m] = d2 * (4.0 * (double)sb.x - g * (double)sa.x);  // alpha^2 = 4
    Mi[m] = d2 * (4.0 * (double)sb.y - g * (double)sa.y);
  }
}

// per-block partial sums of <L:M> and <M:M> (src/RHSfunctions.py:1838-1842).
// kLmBlocks is two CTAs per SM, so the registers are bounded for two: left to
// the compiler the kernel took 172 to 188, one CTA per SM and two waves
// (128^3 FP64 113 us against 82, FP32 70 against 50).
template <typename T>
__global__ void __launch_bounds__(256, 2) dsmag_lm_kernel(const Cx<T>* __restrict__ A, const Cx<T>* __restrict__ B,
                                                       const double* __restrict__ g, int N1, int N2, int N3,
                                                       int n3h, double d2, double* __restrict__ part) {
  const long long fs = (long long)N1 * N2 * n3h;
  const double *g1 = g, *g2 = g + N1, *g3 = g + N1 + N2;
  double num = 0.0, den = 0.0;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < fs; s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % n3h);
    const long long t = s / n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    if (i1 == N1 / 2 || i2 == N2 / 2 || i3 == N3 / 2) continue;  // modes pad() drops
    double Lr[6], Li[6], Mr[6], Mi[6];
    dsmag_lm<T>(A, B, fs, s, g1[i1] * g2[i2] * g3[i3], d2, Lr, Li, Mr, Mi);
    if (i3 > 0) {
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        num += 2.0 * (Lr[m] * Mr[m] + Li[m] * Mi[m]);
        den += 2.0 * (Mr[m] * Mr[m] + Mi[m] * Mi[m]);
      }
    } else {
      // Hermitian part of the k3 = 0 plane: 1/2 Re(L M*) + 1/2 Re(L(k) M(-k))
      const int j1 = (N1 - i1) % N1, j2 = (N2 - i2) % N2;
      const long long sp = ((long long)j1 * N2 + j2) * n3h;
      double pLr[6], pLi[6], pMr[6], pMi[6];
      dsmag_lm<T>(A, B, fs, sp, g1[j1] * g2[j2] * g3[0], d2, pLr, pLi, pMr, pMi);
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        num += 0.5 * (Lr[m] * Mr[m] + Li[m] * Mi[m]) + 0.5 * (Lr[m] * pMr[m] - Li[m] * pMi[m]);
        den += 0.5 * (Mr[m] * Mr[m] + Mi[m] * Mi[m]) + 0.5 * (Mr[m] * pMr[m] - Mi[m] * pMi[m]);
      }
    }
  }
  __shared__ double red[2][256];
  red[0][threadIdx.x] = num;
  red[1][threadIdx.x] = den;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) {
      red[0][threadIdx.x] += red[0][threadIdx.x + h];
      red[1][threadIdx.x] += red[1][threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = red[0][0];
    part[2 * blockIdx.x + 1] = red[1][0];
  }
}

// out[0] = Cs^2 = num/den (IEEE: 0/0 -> NaN, as the reference's np.mean ratio), out[1..2] = num, den
__global__ void __launch_bounds__(256) dsmag_cs2_kernel(const double* __restrict__ part, int nblk,
                                                        double* __restrict__ out) {
  __shared__ double red[2][256];
  double num = 0.0, den = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    num += part[2 * b];
    den += part[2 * b + 1];
  }
  red[0][threadIdx.x] = num;
  red[1][threadIdx.x] = den;
  __syncthreads();
  for (int h = blockDim.x / 2; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) {
      red[0][threadIdx.x] += red[0][threadIdx.x + h];
      red[1][threadIdx.x] += red[1][threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = red[0][0] / red[1][0];
    out[1] = red[0][0];
    out[2] = red[1][0];
  }
}

// the Smagorinsky epilogue on the stored u spectra, tau scaled by -2 Cs^2 Delta^2
template <typename T>
__global__ void __launch_bounds__(256) dsmag_epi_kernel(EpiNS<T, true> epi, const Cx<T>* __restrict__ A, int N1,
                                                        int N2, int n3h, const double* __restrict__ cs2,
                                                        double delta) {
  const long long fs = (long long)N1 * N2 * n3h;
  const T f = (T)(-2.0 * (cs2[0] * delta * delta));
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < fs; s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % n3h);
    const long long t = s / n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    Cx<T> P[12];
#pragma unroll
    for (int m = 0; m < 6; ++m) P[m] = A[m * fs + s];
#pragma unroll
    for (int m = 6; m < 12; ++m) P[m] = f * A[m * fs + s];
    epi(i1, i2, i3, P);
  }
}

// ---------------------------------------------------------------------------
// First-order complete memory model (PySpectral/src/RHSfunctions.py:1411-1542)
// on the state (u, v, w, w0_u, w0_v, w0_w):
//   du/dt  = unpad_2x(PL u) + w0
//   dw0/dt = PLQL u - 250 nu k^2 w0
// PL and PLQL are the t-model's pipelines (run_pl / run_plql, PLQL stored).
// w0_v enters as zero, as in the reference: its Q2U reads it from
// Q[3::6,4::6,4::6] (src/Classes.py:489), a slice nothing writes.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) cm1_combine_kernel(StepIO<T> io, KTabs<T> k, const Cx<T>* __restrict__ PLp,
                                                          const Cx<T>* __restrict__ PLQL, T nu250, int N1, int N2,
                                                          int N3) {
  const long long fs = io.fstride;
  const long long npts = (long long)N1 * N2 * io.n3h;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < npts;
       s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % io.n3h);
    const long long t = s / io.n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    const Cx<T> zero = mk<T>(0, 0);
    const Cx<T> w0u = io.Q[3 * fs + s], w0v = zero, w0w = io.Q[5 * fs + s];
    if (io.read_out) {
      const bool nyq = i1 == N1 / 2 || i2 == N2 / 2 || i3 == N3 / 2;
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * fs + s] = nyq ? zero : io.Q[f * fs + s];
    }
    if (io.w0_out) {
      io.w0_out[s] = w0u;
      io.w0_out[fs + s] = w0v;
      io.w0_out[2 * fs + s] = w0w;
    }
    const T damp = nu250 * ksq;
    const Cx<T> r0 = PLp[s] + w0u, r1 = PLp[fs + s] + w0v, r2 = PLp[2 * fs + s] + w0w;
    const Cx<T> r3 = PLQL[s] - damp * w0u, r4 = PLQL[fs + s] - damp * w0v, r5 = PLQL[2 * fs + s] - damp * w0w;
    io.finish(s, 0, r0);
    io.finish(s, 1, r1);
    io.finish(s, 2, r2);
    io.finish(s, 3, r3);
    io.finish(s, 4, r4);
    io.finish(s, 5, r5);
  }
}

template <typename T>
int cm1_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p) {
  if (p->rotate)
    return fail(c, PSB_ERR_UNSUPPORTED, "PSB_CM1: the reference's computeRHS_CM1 has no rotating form");
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const long long fs = (long long)N1 * N2 * N3h;
  int st = PSB_OK;
  Cx<T>* PLp = scratch<T>(c, "mem.PLp", (size_t)3 * fs, &st);
  Cx<T>* PLQL = scratch<T>(c, "cm1.PLQL", (size_t)3 * fs, &st);
  if (st != PSB_OK) return st;
  const Cx<T>* Qin = io.Q;
  MemCfg m{"memu", nullptr, 0, true, false, 0};
  if (Qin) PSB_TRY(cuda_ok(c, cudaMemsetAsync(PLp, 0, sizeof(Cx<T>) * 3 * fs, c->stream), "memset"));
  Cx<T>*B2 = nullptr, *E = nullptr;
  PSB_TRY(run_pl<T>(c, Qin, p, m, &B2, &E, PLp, nullptr));
  EpiPLQL<T> epi{};
  epi.io = io;
  epi.k = ktabs<T>(c->kx, c->ky, c->kz);
  epi.PLp = PLp;
  epi.coef = (T)0;
  epi.ny1 = N1 / 2;
  epi.ny2 = N2 / 2;
  epi.ny3 = N3 / 2;
  epi.plql_out = PLQL;
  PSB_TRY(run_plql<T>(c, m, Qin ? B2 : nullptr, E, epi));
  if (!Qin) return PSB_OK;  // allocation only
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "cm1 combine", (double)sizeof(Cx<T>) * fs * (6 + 2 + 6));
    cm1_combine_kernel<T><<<blocks, 256, 0, c->stream>>>(io, ktabs<T>(c->kx, c->ky, c->kz), PLp, PLQL,
                                                         (T)(250 * p->nu), N1, N2, N3);
  }
  return launch_ok(c, "cm1 combine");
}

// ---------------------------------------------------------------------------
// First-order finite memory model (PySpectral/src/RHSfunctions.py:882-1024) on
// the state (u, v, w, w0_u^1, w0_v^1, w0_w^1, ..., w0_w^n), n = fm_nsub:
//   du/dt    = unpad_2x(PL u) + sum_i w0^i
//   dw0^i/dt = -2/d w0^i + (-1)^(i+1) 2 PLQL u + S_i,  d = dt0/n,
// S_i = sum_{i'<=i} sum_{j<i'} 4/d (-1)^(i'+j+1) w0^j (the reference's running
// sum is not reset between i).  PL, PLQL: the t-model's pipelines.  With
// rotation the reference adds 2 u x Om to PL on the 2x grid before the mode
// split (:959-962); it is non-zero on the resolved modes only, so PL_q and PLQL
// are unchanged and it joins the velocity RHS.
// ---------------------------------------------------------------------------
constexpr int kFmMaxSub = 8;

template <typename T>
__global__ void __launch_bounds__(256) fm1_combine_kernel(StepIO<T> io, const Cx<T>* __restrict__ PLp,
                                                          const Cx<T>* __restrict__ PLQL, int nsub, T m2d, T p4d,
                                                          int rotate, T Om1, T Om2, T Om3, int N1, int N2, int N3) {
  const long long fs = io.fstride;
  const long long npts = (long long)N1 * N2 * io.n3h;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < npts;
       s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % io.n3h);
    const long long t = s / io.n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    const bool nyq = i1 == N1 / 2 || i2 == N2 / 2 || i3 == N3 / 2;
    Cx<T> ur[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) ur[f] = nyq ? mk<T>(0, 0) : io.Q[f * fs + s];
    if (io.read_out) {
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * fs + s] = ur[f];
    }
    Cx<T> cor[3] = {mk<T>(0, 0), mk<T>(0, 0), mk<T>(0, 0)};
    if (rotate) {
      cor[0] = (T)2 * (Om3 * ur[1] - Om2 * ur[2]);
      cor[1] = (T)2 * (Om1 * ur[2] - Om3 * ur[0]);
      cor[2] = (T)2 * (Om2 * ur[0] - Om1 * ur[1]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<T> w0[kFmMaxSub];
      Cx<T> sum = mk<T>(0, 0);
      for (int i = 0; i < nsub; ++i) {
        w0[i] = io.Q[(3 + 3 * i + c) * fs + s];
        sum = sum + w0[i];
        if (io.w0_out) io.w0_out[(3 * i + c) * fs + s] = w0[i];  // the memory variables as read
      }
      const Cx<T> plql = PLQL[c * fs + s];
      io.finish(s, c, (rotate ? PLp[c * fs + s] + cor[c] : PLp[c * fs + s]) + sum);
      Cx<T> run = mk<T>(0, 0);
      for (int i = 1; i <= nsub; ++i) {
        for (int j = 1; j < i; ++j) run = run + (((i + j + 1) & 1) ? -p4d : p4d) * w0[j - 1];
        const T sgn2 = ((i + 1) & 1) ? (T)-2 : (T)2;
        io.finish(s, 3 + 3 * (i - 1) + c, (m2d * w0[i - 1] + sgn2 * plql) + run);
      }
    }
  }
}

template <typename T>
int fm1_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p) {
  const int nsub = p->fm_nsub > 0 ? p->fm_nsub : 1;
  if (nsub > kFmMaxSub) return fail(c, PSB_ERR_ARG, "PSB_FM1: fm_nsub must be 1..8");
  const double dt0 = p->fm_dt0 > 0 ? p->fm_dt0 : 0.1;
  const double d = dt0 / nsub;
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const long long fs = (long long)N1 * N2 * N3h;
  int st = PSB_OK;
  Cx<T>* PLp = scratch<T>(c, "mem.PLp", (size_t)3 * fs, &st);
  Cx<T>* PLQL = scratch<T>(c, "fm1.PLQL", (size_t)3 * fs, &st);
  if (st != PSB_OK) return st;
  const Cx<T>* Qin = io.Q;
  MemCfg m{"memu", nullptr, 0, true, false, 0};
  if (Qin) PSB_TRY(cuda_ok(c, cudaMemsetAsync(PLp, 0, sizeof(Cx<T>) * 3 * fs, c->stream), "memset"));
  Cx<T>*B2 = nullptr, *E = nullptr;
  PSB_TRY(run_pl<T>(c, Qin, p, m, &B2, &E, PLp, nullptr));
  EpiPLQL<T> epi{};
  epi.io = io;
  epi.k = ktabs<T>(c->kx, c->ky, c->kz);
  epi.PLp = PLp;
  epi.coef = (T)0;
  epi.ny1 = N1 / 2;
  epi.ny2 = N2 / 2;
  epi.ny3 = N3 / 2;
  epi.plql_out = PLQL;
  PSB_TRY(run_plql<T>(c, m, Qin ? B2 : nullptr, E, epi));
  if (!Qin) return PSB_OK;  // allocation only
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "fm1 combine", (double)sizeof(Cx<T>) * fs * (3 + 3 * nsub) * 2 + sizeof(Cx<T>) * fs * 6);
    fm1_combine_kernel<T><<<blocks, 256, 0, c->stream>>>(io, PLp, PLQL, nsub, (T)(-2. / d), (T)(4. / d), p->rotate,
                                                         (T)p->Om1, (T)p->Om2, (T)p->Om3, N1, N2, N3);
  }
  return launch_ok(c, "fm1 combine");
}

// ---------------------------------------------------------------------------
// Second-order finite memory model (PySpectral/src/RHSfunctions.py:1025-1286,
// turb_model 4; setup src/Classes.py:294-401).  State: u, then per
// subintegration i the pairs w0^i (fields 3 + 6i) and w1^i (fields 6 + 6i)
// (the interleaved layout of src/Classes.py:330-355 with equal numbers of w0
// and w1 subintegrations).  One RHS =
//   A  u -> PL on the whole 2x grid (kept), its q part and unpad_2x(PL);
//   B  u_j (PL_q)_i -> PLQL on the whole 2x grid: its q part (2x grid),
//      unpad_2x(PLQL) and unpad_2x(PLQL_q) (N grid);
//   C  PL_a (PL_q)_b on the 3N grid (pad() of the 2x grid), truncated to the
//      N grid (unpad_2x(unpad(.)), :1168-1186);
//   D  (PLQL_q)_i u_j on the 2x grid, truncated to the N grid (:1188-1204);
//   E  one kernel: pterm, pterm2, PLQLQL (:1206-1224) and the memory
//      equations (:1236-1282), fused with the RK stage update.
// ---------------------------------------------------------------------------

// Stage C: nine products PL_a (PL_q)_b of two 3-field sets given on the whole
// 2x grid (3, 2N1, 2N2, N3+1): pad() to the 3N grid (drops the 2x grid's
// index N of x and y and its k3 = N plane, src/padding.py:16-25), c2r scaled
// by sqrt(3^3 sqrt(N1 N2 N3)) (:1155), products, r2c, and unpad() then
// unpad_2x() straight to the N grid: N-grid row i < N/2 comes from 3N-grid row
// i, row i >= N/2 from row i + 2N; k3 < N3/2.  out9: (9, N1, N2, N3/2+1),
// product 3a + b = PL_a (PL_q)_b; its k3 = N3/2 plane is written zero.
template <typename T>
int run_fm2_3n(psb_ctx* c, const Cx<T>* PL, const Cx<T>* PLq, Cx<T>* out9) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int F1 = 2 * N1, F2 = 2 * N2, F3h = N3 + 1;
  const int M1 = 3 * N1, M2 = 3 * N2, M3 = 3 * N3, Kz = N3, Ko = N3 / 2;
  int st = PSB_OK;
  Cx<T>* A = scratch<T>(c, "fm2.A3n", (size_t)6 * M1 * F2 * Kz, &st);
  Cx<T>* B = scratch<T>(c, "fm2.B3n", (size_t)6 * M1 * M2 * Kz, &st);
  Cx<T>* C = scratch<T>(c, "fm2.C3n", (size_t)9 * M1 * M2 * Ko, &st);
  Cx<T>* D = scratch<T>(c, "fm2.D3n", (size_t)9 * M1 * N2 * Ko, &st);
  if (st != PSB_OK) return st;
  if (!PL) return PSB_OK;  // allocation only
  const long long fsC = (long long)F1 * F2 * F3h, fsA = (long long)M1 * F2 * Kz;
  const psb::RowMap to3n1 = psb::RowMap{N1, N1 + 1, N1}, to3n2 = psb::RowMap{N2, N2 + 1, N2};
  for (int set = 0; set < 2; ++set) {
    AxisArgs<T> a = axis_common<T>(c, M1);
    a.in = set == 0 ? PL : PLq;
    a.out = A + set * 3 * fsA;
    a.in_fstride = fsC;
    a.in_ostride = F3h;
    a.in_rstride = (long long)F2 * F3h;
    a.out_fstride = fsA;
    a.out_ostride = Kz;
    a.out_rstride = (long long)F2 * Kz;
    a.nouter = F2;
    a.ncols = Kz;
    a.in_rows = F1;
    a.out_rows = M1;
    a.in_map = to3n1;
    a.out_map = map_id(M1);
    PSB_TRY((launch_axis<T, true>(c, a, PreCopyN<T, 3>{}, "3n x-inverse")));
  }
  AxisArgs<T> b = axis_common<T>(c, M2);
  b.in = A;
  b.out = B;
  b.in_ostride = (long long)F2 * Kz;
  b.in_rstride = Kz;
  b.out_ostride = (long long)M2 * Kz;
  b.out_rstride = Kz;
  b.nouter = 6 * M1;
  b.ncols = Kz;
  b.in_rows = F2;
  b.out_rows = M2;
  b.in_map = to3n2;
  b.out_map = map_id(M2);
  const double s3 = std::sqrt(27.0 * std::sqrt((double)N1 * N2 * N3));
  const double fac = s3 / ((double)M1 * M2 * M3), fsc = field_scale(fac);
  b.scale = (T)fsc;
  PSB_TRY((launch_axis<T, true>(c, b, PreCopy<T>{}, "3n y-inverse")));
  ZArgs<T> z{};
  const long long fsB = (long long)M1 * M2 * Kz, fsO = (long long)M1 * M2 * Ko;
  for (int f = 0; f < 6; ++f) {
    z.in[f] = B + f * fsB;
    z.in_pstride[f] = Kz;
    z.in_kz[f] = Kz;
  }
  for (int g = 0; g < 9; ++g) {
    z.out[g] = C + g * fsO;
    z.out_pstride[g] = Ko;
  }
  z.out_kz = Ko;
  z.npencils = (long long)M1 * M2;
  z.fac = (T)(fac / fsc);
  z.plan = *plan_for(c, M3);
  z.tw = twiddles<T>(c);
  PSB_TRY(launch_z<T>(c, z, PhysPLQL<T>{}, "3n z-products"));
  AxisArgs<T> d = axis_common<T>(c, M2);
  d.in = C;
  d.out = D;
  d.in_ostride = (long long)M2 * Ko;
  d.in_rstride = Ko;
  d.out_ostride = (long long)N2 * Ko;
  d.out_rstride = Ko;
  d.nouter = 9 * M1;
  d.ncols = Ko;
  d.in_rows = M2;
  d.out_rows = N2;
  d.in_map = map_id(M2);
  d.out_map = psb::RowMap{N2 / 2, N2 / 2, 2 * N2};
  PSB_TRY((launch_axis<T, false>(c, d, PreCopy<T>{}, "3n y-forward")));
  XEpiArgs<T> e{};
  e.in = D;
  e.in_fstride = (long long)M1 * N2 * Ko;
  e.in_rstride = (long long)N2 * Ko;
  e.in_ostride = Ko;
  e.n1 = N1;
  e.n2 = N2;
  e.n3h = N3h;
  e.kz = Ko;
  e.out_map = psb::RowMap{N1 / 2, N1 / 2, 2 * N1};
  e.plan = *plan_for(c, M1);
  e.tw = twiddles<T>(c);
  return launch_epi<T>(c, e, EpiStore<T, 9>{out9, (long long)N1 * N2 * N3h, N2, N3h}, "3n x-forward+store");
}

// Stage E: PLQLQL and every right-hand side of the state, with the RK stage
// update.  P3[3a + b] = PL_a (PL_q)_b, P2[3j + i] = (PLQL_q)_i u_j (N grid).
template <typename T>
__global__ void __launch_bounds__(256) fm2_combine_kernel(StepIO<T> io, KTabs<T> k, const Cx<T>* __restrict__ PLp,
                                                          const Cx<T>* __restrict__ PLQL,
                                                          const Cx<T>* __restrict__ PLQLq,
                                                          const Cx<T>* __restrict__ P3, const Cx<T>* __restrict__ P2,
                                                          int nsub, T nu, T m2d0, T p4d0, T m2d1, T p4d1, int N1,
                                                          int N2, int N3) {
  const long long fs = io.fstride;
  const long long npts = (long long)N1 * N2 * io.n3h;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < npts;
       s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % io.n3h);
    const long long t = s / io.n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    if (io.read_out) {
      const bool nyq = i1 == N1 / 2 || i2 == N2 / 2 || i3 == N3 / 2;
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * fs + s] = nyq ? mk<T>(0, 0) : io.Q[f * fs + s];
    }
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    Cx<T> A[9], B[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) {
      A[m] = P3[m * fs + s];
      B[m] = P2[m * fs + s];
    }
    // names of the reference: A = PLa_PLbq at 3a + b, B = PLQLiq_jp at 3j + i
    const Cx<T> uu = A[0], uv = A[1], uw = A[2], vu = A[3], vv = A[4], vw = A[5], wu = A[6], wv = A[7], ww = A[8];
    const Cx<T> qu_u = B[0], qv_u = B[1], qw_u = B[2], qu_v = B[3], qv_v = B[4], qw_v = B[5], qu_w = B[6],
                qv_w = B[7], qw_w = B[8];
    const Cx<T> pterm = ksqi * ((k1 * k1) * uu + (k2 * k2) * vv + (k3 * k3) * ww + (k1 * k2) * (vu + uv) +
                                (k1 * k3) * (uw + wu) + (k2 * k3) * (vw + wv));
    const Cx<T> pterm2 = ksqi * ((k1 * k1) * qu_u + (k2 * k2) * qv_v + (k3 * k3) * qw_w + (k1 * k2) * (qv_u + qu_v) +
                                 (k1 * k3) * (qw_u + qu_w) + (k2 * k3) * (qw_v + qv_w));
    const T two = (T)2;
    const Cx<T> QQ[3] = {
        mik(two * k1, uu) + mik(k2, vu) + mik(k3, wu) + mik(k2, uv) + mik(k3, uw) + pik(two * k1, pterm) +
            pik(two * k1, qu_u) + mik(k2, qv_u) + mik(k3, qw_u) + mik(k2, qu_v) + mik(k3, qu_w) +
            pik(two * k1, pterm2) - (nu * ksq) * PLQLq[s],
        mik(k1, uv) + mik(two * k2, vv) + mik(k3, wv) + mik(k1, vu) + mik(k3, vw) + pik(two * k2, pterm) +
            mik(k1, qu_v) + mik(two * k2, qv_v) + mik(k3, qw_v) + mik(k1, qv_u) + mik(k3, qv_w) +
            pik(two * k2, pterm2) - (nu * ksq) * PLQLq[fs + s],
        mik(k1, uw) + mik(k2, vw) + mik(two * k3, ww) + mik(k1, wu) + mik(k2, wv) + pik(two * k3, pterm) +
            mik(k1, qu_w) + mik(k2, qv_w) + mik(two * k3, qw_w) + mik(k1, qw_u) + mik(k3, qw_v) +
            pik(two * k3, pterm2) - (nu * ksq) * PLQLq[2 * fs + s]};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<T> w0[kFmMaxSub], w1[kFmMaxSub];
      Cx<T> sum = mk<T>(0, 0);
      for (int i = 0; i < nsub; ++i) {
        w0[i] = io.Q[(3 + 6 * i + c) * fs + s];
        w1[i] = io.Q[(6 + 6 * i + c) * fs + s];
        sum = sum + w0[i];
        if (io.w0_out) {  // the memory variables as read (main.w0_*, main.w1_*)
          io.w0_out[(6 * i + c) * fs + s] = w0[i];
          io.w0_out[(6 * i + 3 + c) * fs + s] = w1[i];
        }
      }
      io.finish(s, c, PLp[c * fs + s] + sum);
      const Cx<T> plql = PLQL[c * fs + s];
      Cx<T> run0 = mk<T>(0, 0), run1 = mk<T>(0, 0);
      for (int i = 1; i <= nsub; ++i) {
        for (int j = 1; j < i; ++j) {
          const bool neg = ((i + j + 1) & 1) != 0;
          run0 = run0 + (neg ? -p4d0 : p4d0) * w0[j - 1];
          run1 = run1 + (neg ? -p4d1 : p4d1) * w1[j - 1];
        }
        const T sgn2 = ((i + 1) & 1) ? (T)-2 : (T)2;
        io.finish(s, 3 + 6 * (i - 1) + c, ((m2d0 * w0[i - 1] + sgn2 * plql) + run0) + w1[i - 1]);
        io.finish(s, 6 + 6 * (i - 1) + c, (m2d1 * w1[i - 1] + sgn2 * QQ[c]) + run1);
      }
    }
  }
}

template <typename T>
int fm2_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p) {
  if (p->rotate) return fail(c, PSB_ERR_UNSUPPORTED, "PSB_FM2: the reference has no rotating form");
  const int nsub = p->fm_nsub > 0 ? p->fm_nsub : 1;
  if (nsub > kFmMaxSub) return fail(c, PSB_ERR_ARG, "PSB_FM2: fm_nsub must be 1..8");
  // the 3N-grid passes hold one 3N-point line per field in shared memory
  if (3 * std::max(c->N1, std::max(c->N2, c->N3)) > (c->prec == 64 ? 768 : 1536))
    return fail(c, PSB_ERR_SHAPE, "PSB_FM2: grid too large for the 3N-grid products (N <= 256 FP64, 512 FP32)");
  const double d0 = (p->fm_dt0 > 0 ? p->fm_dt0 : 0.1) / nsub;
  const double d1 = (p->fm_dt1 > 0 ? p->fm_dt1 : 0.05) / nsub;
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const long long fs = (long long)N1 * N2 * N3h;
  const long long fs2 = (long long)2 * N1 * 2 * N2 * (N3 + 1);
  int st = PSB_OK;
  Cx<T>* PLp = scratch<T>(c, "mem.PLp", (size_t)3 * fs, &st);
  Cx<T>* PLfull = scratch<T>(c, "fm2.PL", (size_t)3 * fs2, &st);
  Cx<T>* PLQLq2 = scratch<T>(c, "fm2.PLQLq2", (size_t)3 * fs2, &st);
  Cx<T>* N6 = scratch<T>(c, "fm2.PLQLn", (size_t)6 * fs, &st);  // unpad_2x(PLQL), unpad_2x(PLQL_q)
  Cx<T>* P3 = scratch<T>(c, "fm2.P3", (size_t)9 * fs, &st);
  Cx<T>* P2 = scratch<T>(c, "fm2.P2", (size_t)9 * fs, &st);
  if (st != PSB_OK) return st;
  const Cx<T>* Qin = io.Q;
  MemCfg m{"memu", nullptr, 0, true, false, 0};
  if (Qin) {
    PSB_TRY(cuda_ok(c, cudaMemsetAsync(PLp, 0, sizeof(Cx<T>) * 3 * fs, c->stream), "memset"));
    PSB_TRY(cuda_ok(c, cudaMemsetAsync(N6, 0, sizeof(Cx<T>) * 6 * fs, c->stream), "memset"));
  }
  Cx<T>*B2 = nullptr, *E = nullptr;
  PSB_TRY(run_pl<T>(c, Qin, p, m, &B2, &E, PLp, nullptr, PLfull));
  EpiPLQLFull<T> ef{};
  ef.kf = ktabs<T>(c->kxf, c->kyf, c->kzf);
  ef.N1 = N1;
  ef.N2 = N2;
  ef.N3 = N3;
  ef.n3h = N3h;
  ef.nf2 = 2 * N2;
  ef.nf3h = N3 + 1;
  ef.fstride_2x = fs2;
  ef.fstride_n = fs;
  ef.PLQLq = PLQLq2;
  ef.PLQLn = N6;
  ef.PLQLqn = N6 + 3 * fs;
  PSB_TRY((run_plql<T, EpiPLQLFull<T>, true>(c, m, Qin ? B2 : nullptr, E, ef)));
  PSB_TRY(run_fm2_3n<T>(c, Qin ? PLfull : nullptr, E, P3));
  PSB_TRY((run_plql<T, EpiStore<T, 9>>(c, m, Qin ? B2 : nullptr, PLQLq2, EpiStore<T, 9>{P2, fs, N2, N3h})));
  if (!Qin) return PSB_OK;  // allocation only
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "fm2 combine",
                   (double)sizeof(Cx<T>) * fs * ((3 + 6 * nsub) * 2 + 3 + 6 + 18 + (io.read_out ? 3 : 0)));
    fm2_combine_kernel<T><<<blocks, 256, 0, c->stream>>>(io, ktabs<T>(c->kx, c->ky, c->kz), PLp, N6, N6 + 3 * fs,
                                                         P3, P2, nsub, (T)p->nu, (T)(-2. / d0), (T)(4. / d0),
                                                         (T)(-2. / d1), (T)(4. / d1), N1, N2, N3);
  }
  return launch_ok(c, "fm2 combine");
}

// ---------------------------------------------------------------------------
// DNS with SGS budgets (PySpectral/src/RHSfunctions.py:1543-1661, turb_model 99):
// RHS = unpad_2x(PL u); PLQL u with the q part split at main.kc
// (seperateModesBudgets, src/padding.py:81-93) is stored for the budget files.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) budgets_finish_kernel(StepIO<T> io, const Cx<T>* __restrict__ PLp, int N1,
                                                             int N2, int N3) {
  const long long fs = io.fstride;
  const long long npts = (long long)N1 * N2 * io.n3h;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < npts;
       s += (long long)gridDim.x * blockDim.x) {
    if (io.read_out) {
      const int i3 = (int)(s % io.n3h);
      const long long t = s / io.n3h;
      const int i2 = (int)(t % N2), i1 = (int)(t / N2);
      const bool nyq = i1 == N1 / 2 || i2 == N2 / 2 || i3 == N3 / 2;
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * fs + s] = nyq ? mk<T>(0, 0) : io.Q[f * fs + s];
    }
    io.finish(s, 0, PLp[s]);
    io.finish(s, 1, PLp[fs + s]);
    io.finish(s, 2, PLp[2 * fs + s]);
  }
}

template <typename T>
int budgets_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p) {
  if (p->rotate)
    return fail(c, PSB_ERR_UNSUPPORTED, "PSB_BUDGETS: the reference's computeRHS_BUDGETS has no rotating form");
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const long long fs = (long long)N1 * N2 * N3h;
  // main.kc = amax(grid.k1) (src/Classes.py:16), truncated by the slices of seperateModesBudgets
  const int kc = p->kf > 0 ? p->kf : (int)(((double)(N1 / 2 - 1) * 2.0) * M_PI / c->L1);
  if (kc < 2 || kc > N1 || kc > N2 || kc > N3 / 2 + 1)
    return fail(c, PSB_ERR_ARG, "PSB_BUDGETS: budget split kc (p.kf) out of range");
  int st = PSB_OK;
  Cx<T>* PLp = scratch<T>(c, "mem.PLp", (size_t)3 * fs, &st);
  Cx<T>* PLQL = io.w0_out ? io.w0_out : scratch<T>(c, "budget.PLQL", (size_t)3 * fs, &st);
  if (st != PSB_OK) return st;
  const Cx<T>* Qin = io.Q;
  MemCfg m{"memu", nullptr, kc, true, false, 0};
  if (Qin) PSB_TRY(cuda_ok(c, cudaMemsetAsync(PLp, 0, sizeof(Cx<T>) * 3 * fs, c->stream), "memset"));
  Cx<T>*B2 = nullptr, *E = nullptr;
  PSB_TRY(run_pl<T>(c, Qin, p, m, &B2, &E, PLp, nullptr));
  EpiPLQL<T> epi{};
  epi.io = io;
  epi.k = ktabs<T>(c->kx, c->ky, c->kz);
  epi.PLp = PLp;
  epi.coef = (T)0;
  epi.ny1 = N1 / 2;
  epi.ny2 = N2 / 2;
  epi.ny3 = N3 / 2;
  epi.plql_out = PLQL;
  PSB_TRY(run_plql<T>(c, m, Qin ? B2 : nullptr, E, epi));
  if (!Qin) return PSB_OK;  // allocation only
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "budgets finish", (double)sizeof(Cx<T>) * fs * (3 + 3 + 3));
    budgets_finish_kernel<T><<<blocks, 256, 0, c->stream>>>(io, PLp, N1, N2, N3);
  }
  return launch_ok(c, "budgets finish");
}

// ---------------------------------------------------------------------------
// Orthogonal dynamics (PySpectral/src/RHSfunctions.py:53-143): the DNS RHS of u
// minus the DNS RHS of Gf u, each with its own pressure and Coriolis terms.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ Cx<T> ortho_part(T k1, T k2, T k3, T ksq, T ksqi, T nu, const Cx<T>* P, const Cx<T>* u,
                                            int comp, int rotate, T Om1, T Om2, T Om3, Cx<T>* cor) {
  const Cx<T> uu = P[0], vv = P[1], ww = P[2], uv = P[3], uw = P[4], vw = P[5];
  Cx<T> ph = ksqi * ((-k1 * k1) * uu - (k2 * k2) * vv - (k3 * k3) * ww - ((T)2 * k1 * k2) * uv -
                     ((T)2 * k1 * k3) * uw - ((T)2 * k2 * k3) * vw);
  const Cx<T> cu = Om3 * u[1] - Om2 * u[2], cv = Om1 * u[2] - Om3 * u[0], cw = Om2 * u[0] - Om1 * u[1];
  if (rotate) ph = ph - ((T)2 * ksqi) * mul_i(k1 * cu + k2 * cv + k3 * cw);
  const Cx<T> c3[3] = {cu, cv, cw};
  *cor = (T)2 * c3[comp];
  if (comp == 0) return mik(k1, uu) + mik(k2, uv) + mik(k3, uw) + mik(k1, ph) - (nu * ksq) * u[0];
  if (comp == 1) return mik(k1, uv) + mik(k2, vv) + mik(k3, vw) + mik(k2, ph) - (nu * ksq) * u[1];
  return mik(k1, uw) + mik(k2, vw) + mik(k3, ww) + mik(k3, ph) - (nu * ksq) * u[2];
}

template <typename T>
__global__ void __launch_bounds__(256) ortho_combine_kernel(StepIO<T> io, KTabs<T> k, const Cx<T>* __restrict__ A,
                                                            const Cx<T>* __restrict__ B, const double* __restrict__ gx,
                                                            const double* __restrict__ gy,
                                                            const double* __restrict__ gz, T nu, int rotate, T Om1,
                                                            T Om2, T Om3, int N1, int N2, int N3) {
  const long long fs = io.fstride;
  const long long npts = (long long)N1 * N2 * io.n3h;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < npts;
       s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % io.n3h);
    const long long t = s / io.n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    const bool nyq = i1 == N1 / 2 || i2 == N2 / 2 || i3 == N3 / 2;
    const T gf = (T)(gx[i1] * gy[i2] * gz[i3]);
    Cx<T> u[3], uf[3], P[6], Pf[6];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      u[f] = nyq ? mk<T>(0, 0) : io.Q[f * fs + s];
      uf[f] = gf * u[f];
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      P[m] = A[m * fs + s];
      Pf[m] = B[m * fs + s];
    }
    if (io.read_out) {
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * fs + s] = u[f];
    }
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    Cx<T> R[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<T> cor, corf;
      const Cx<T> a = ortho_part(k1, k2, k3, ksq, ksqi, nu, P, u, c, rotate, Om1, Om2, Om3, &cor);
      const Cx<T> af = ortho_part(k1, k2, k3, ksq, ksqi, nu, Pf, uf, c, rotate, Om1, Om2, Om3, &corf);
      Cx<T> r = rotate ? a + cor : a;
      r = r - af;
      R[c] = rotate ? r - corf : r;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) io.finish(s, c, R[c]);
  }
}

template <typename T>
int ortho_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p, const psb_tuned* ts) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const long long fs = (long long)N1 * N2 * N3h;
  int st = PSB_OK;
  Cx<T>* A = scratch<T>(c, "ortho.A", (size_t)6 * fs, &st);
  Cx<T>* B = scratch<T>(c, "ortho.B", (size_t)6 * fs, &st);
  if (st != PSB_OK) return st;
  const Cx<T>* Qin = io.Q;
  EpiStore<T, 6> sa{A, fs, N2, N3h}, sb{B, fs, N2, N3h};
  PSB_TRY(run_ns32<T>(c, Qin, PreCopyN<T, 3>{}, PhysProducts<T>{}, sa, ts));
  PSB_TRY(run_ns32<T>(c, Qin, PreMask3<T>{c->gx, c->gy, c->gz}, PhysProducts<T>{}, sb, ts));
  if (!Qin) return PSB_OK;  // allocation only
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "ortho combine", (double)sizeof(Cx<T>) * fs * (12 + 3) + io.bytes(fs, 3));
    ortho_combine_kernel<T><<<blocks, 256, 0, c->stream>>>(io, ktabs<T>(c->kx, c->ky, c->kz), A, B, c->gx, c->gy,
                                                           c->gz, (T)p->nu, p->rotate, (T)p->Om1, (T)p->Om2,
                                                           (T)p->Om3, N1, N2, N3);
  }
  return launch_ok(c, "ortho combine");
}

// ---------------------------------------------------------------------------
// Navier-Stokes of the MPI solver (PySpectral/src_MPI/RHSfunctions.py:22-93)
// and its orthogonal dynamics (:179-268): 2/3-rule masks D on read and on the
// RHS, products on the N grid (the MHD pipeline's passes, run_n23).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ Cx<T> mpi_ns_part(T k1, T k2, T k3, T ksq, T ksqi, T nu, T D, const Cx<T>* P,
                                             const Cx<T>* u, int comp, int rotate, T Om1, T Om2, T Om3, Cx<T>* cor) {
  const Cx<T> ph0 = ksqi * ((-k1 * k1) * P[0] - (k2 * k2) * P[1] - (k3 * k3) * P[2] - ((T)2 * k1 * k2) * P[3] -
                            ((T)2 * k1 * k3) * P[4] - ((T)2 * k2 * k3) * P[5]);
  const Cx<T> cu = Om3 * u[1] - Om2 * u[2], cv = Om1 * u[2] - Om3 * u[0], cw = Om2 * u[0] - Om1 * u[1];
  const Cx<T> ph = rotate ? ph0 - ((T)2 * ksqi) * mul_i(k1 * cu + k2 * cv + k3 * cw) : ph0;
  const Cx<T> c3[3] = {cu, cv, cw};
  *cor = (T)2 * c3[comp];
  if (comp == 0) return D * (mik(k1, P[0]) + mik(k2, P[3]) + mik(k3, P[4]) + mik(k1, ph) - (nu * ksq) * u[0]);
  if (comp == 1) return D * (mik(k1, P[3]) + mik(k2, P[1]) + mik(k3, P[5]) + mik(k2, ph) - (nu * ksq) * u[1]);
  return D * (mik(k1, P[4]) + mik(k2, P[5]) + mik(k3, P[2]) + mik(k3, ph) - (nu * ksq) * u[2]);
}

template <typename T>
struct EpiMpiNS {
  static constexpr int F_IN = 6;
  __host__ double io_bytes(long long npts) const { return io.bytes(npts, 3); }
  StepIO<T> io;
  KTabs<T> k;
  const double *m1, *m2, *m3;
  T nu;
  int rotate;
  T Om1, Om2, Om3;
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const {
    const long long s = io.sidx(i1, i2, i3);
    const T D = (T)(m1[i1] * m2[i2] * m3[i3]);
    Cx<T> u[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) u[f] = D * io.Q[f * io.fstride + s];
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    if (io.read_out) {
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * io.fstride + s] = u[f];
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<T> cor;
      const Cx<T> r = mpi_ns_part(k1, k2, k3, ksq, ksqi, nu, D, P, u, c, rotate, Om1, Om2, Om3, &cor);
      io.finish(s, c, rotate ? r + cor : r);
    }
  }
};

// the 2/3 mask and then grid.filter (src_MPI/Classes.py:219-235) on load
template <typename T>
struct PreMask3x2 {
  static constexpr int F_SRC = 3, F_DST = 3;
  const double *m1, *m2, *m3, *f1, *f2, *f3;
  __device__ void operator()(int i, int o, int cc, const AxisArgs<T>&, const Cx<T>* s, Cx<T>* d) const {
    const T m = (T)(m1[i] * m2[o] * m3[cc]), f = (T)(f1[i] * f2[o] * f3[cc]);
#pragma unroll
    for (int q = 0; q < 3; ++q) d[q] = f * (m * s[q]);
  }
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t = copy_fields<T>(3, m1, m2, m3);
    t.f1 = f1;
    t.f2 = f2;
    t.f3 = f3;
    return t;
  }
};

template <typename T>
__global__ void __launch_bounds__(256) mpi_ortho_combine_kernel(StepIO<T> io, KTabs<T> k,
                                                                const Cx<T>* __restrict__ A,
                                                                const Cx<T>* __restrict__ B, const double* __restrict__ m1,
                                                                const double* __restrict__ m2,
                                                                const double* __restrict__ m3,
                                                                const double* __restrict__ gx,
                                                                const double* __restrict__ gy,
                                                                const double* __restrict__ gz, T nu, int rotate, T Om1,
                                                                T Om2, T Om3, int N1, int N2) {
  const long long fs = io.fstride;
  const long long npts = (long long)N1 * N2 * io.n3h;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < npts;
       s += (long long)gridDim.x * blockDim.x) {
    const int i3 = (int)(s % io.n3h);
    const long long t = s / io.n3h;
    const int i2 = (int)(t % N2), i1 = (int)(t / N2);
    const T D = (T)(m1[i1] * m2[i2] * m3[i3]);
    const T gf = (T)(gx[i1] * gy[i2] * gz[i3]);
    Cx<T> u[3], uf[3], P[6], Pf[6];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      u[f] = D * io.Q[f * fs + s];
      uf[f] = gf * u[f];
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      P[m] = A[m * fs + s];
      Pf[m] = B[m * fs + s];
    }
    if (io.read_out) {
#pragma unroll
      for (int f = 0; f < 3; ++f) io.read_out[f * fs + s] = u[f];
    }
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    Cx<T> R[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<T> cor, corf;
      const Cx<T> a = mpi_ns_part(k1, k2, k3, ksq, ksqi, nu, D, P, u, c, rotate, Om1, Om2, Om3, &cor);
      const Cx<T> af = mpi_ns_part(k1, k2, k3, ksq, ksqi, nu, D, Pf, uf, c, rotate, Om1, Om2, Om3, &corf);
      Cx<T> r = rotate ? a + cor : a;
      r = r - af;
      R[c] = rotate ? r - corf : r;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) io.finish(s, c, R[c]);
  }
}

// One semi-implicit step of the MPI solver's Navier-Stokes
// (src_MPI/time_schemes.py:9-11 with the 'Semi-Implicit' branch of
// computeRHS_NOSGS, src_MPI/RHSfunctions.py:70-93): H = the masked nonlinear
// term (+ Coriolis), then
//   Q <- (Q + dt/2 (3 H - H_old) + dt/2 (-nu k^2 u)) / (1 + nu dt/2 k^2)
// with u the masked state; H holds H_old on entry and H on exit.
template <typename T>
struct EpiMpiSI {
  static constexpr int F_IN = 6;
  __host__ double io_bytes(long long npts) const { return (double)sizeof(Cx<T>) * npts * 3 * 5; }
  Cx<T>* Q;
  Cx<T>* H;
  Cx<T>* read_out;
  long long fstride;
  int n2, n3h;
  KTabs<T> k;
  const double *m1, *m2, *m3;
  T nu, dt;
  int rotate;
  T Om1, Om2, Om3;
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const {
    const long long s = ((long long)i1 * n2 + i2) * n3h + i3;
    const T D = (T)(m1[i1] * m2[i2] * m3[i3]);
    Cx<T> q[3], u[3];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      q[f] = Q[f * fstride + s];
      u[f] = D * q[f];
    }
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    const T half = dt / (T)2, den = (T)1 + ((nu * dt) / (T)2) * ksq;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cx<T> cor;
      Cx<T> h = mpi_ns_part(k1, k2, k3, ksq, ksqi, (T)0, D, P, u, c, rotate, Om1, Om2, Om3, &cor);
      if (rotate) h = h + cor;
      const Cx<T> hold = H[c * fstride + s];
      const Cx<T> visc = (-nu * ksq) * u[c];
      const Cx<T> num = (q[c] + half * ((T)3 * h - hold)) + half * visc;
      Q[c * fstride + s] = mk<T>(num.x / den, num.y / den);
      H[c * fstride + s] = h;
      if (read_out) read_out[c * fstride + s] = u[c];
    }
  }
};

template <typename T>
int mpi_si_step(psb_ctx* c, Cx<T>* Q, Cx<T>* H, Cx<T>* read_out, const psb_params* p) {
  EpiMpiSI<T> epi{Q, H, read_out, (long long)c->N1 * c->N2 * c->N3h, c->N2, c->N3h, ktabs<T>(c->kx, c->ky, c->kz),
                  c->mx, c->my, c->mz, (T)p->nu, (T)p->dt, p->rotate, (T)p->Om1, (T)p->Om2, (T)p->Om3};
  return run_n23<T>(c, Q, PreMask3<T>{c->mx, c->my, c->mz}, PhysProducts<T>{}, epi);
}

template <typename T>
int mpi_ns_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p, bool ortho) {
  const int N1 = c->N1, N2 = c->N2, N3h = c->N3h;
  const Cx<T>* Qin = io.Q;
  if (!ortho) {
    EpiMpiNS<T> epi{io, ktabs<T>(c->kx, c->ky, c->kz), c->mx, c->my, c->mz, (T)p->nu, p->rotate,
                    (T)p->Om1, (T)p->Om2, (T)p->Om3};
    return run_n23<T>(c, Qin, PreMask3<T>{c->mx, c->my, c->mz}, PhysProducts<T>{}, epi);
  }
  const long long fs = (long long)N1 * N2 * N3h;
  int st = PSB_OK;
  Cx<T>* A = scratch<T>(c, "mpio.A", (size_t)6 * fs, &st);
  Cx<T>* B = scratch<T>(c, "mpio.B", (size_t)6 * fs, &st);
  if (st != PSB_OK) return st;
  EpiStore<T, 6> sa{A, fs, N2, N3h}, sb{B, fs, N2, N3h};
  PSB_TRY(run_n23<T>(c, Qin, PreMask3<T>{c->mx, c->my, c->mz}, PhysProducts<T>{}, sa));
  PSB_TRY(run_n23<T>(c, Qin, PreMask3x2<T>{c->mx, c->my, c->mz, c->gx, c->gy, c->gz}, PhysProducts<T>{}, sb));
  if (!Qin) return PSB_OK;  // allocation only
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "mpi ortho combine", (double)sizeof(Cx<T>) * fs * 12 + io.bytes(fs, 3));
    mpi_ortho_combine_kernel<T><<<blocks, 256, 0, c->stream>>>(io, ktabs<T>(c->kx, c->ky, c->kz), A, B, c->mx,
                                                               c->my, c->mz, c->gx, c->gy, c->gz, (T)p->nu, p->rotate,
                                                               (T)p->Om1, (T)p->Om2, (T)p->Om3, N1, N2);
  }
  return launch_ok(c, "mpi ortho combine");
}

// myFilter's kept rows (src/Classes.py:1271-1279) with Python slice bounds:
// [0:kc] and [-kc+1:] on axes 1 and 2, [0:kc] on axis 3
inline void myfilter_rows(int n, int kc, bool two_sided, double* out) {
  for (int i = 0; i < n; ++i) out[i] = 0.0;
  for (int i = 0; i < std::min(kc, n); ++i) out[i] = 1.0;
  if (!two_sided) return;
  int lo = 1 - kc;
  if (lo < 0) lo += n;
  lo = std::max(0, std::min(lo, n));
  for (int i = lo; i < n; ++i) out[i] = 1.0;
}

template <typename T>
int dsmag_rhs(psb_ctx* c, StepIO<T> io, const psb_params* p, const psb_tuned* ts, double* cs2_out) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const long long fs = (long long)N1 * N2 * N3h;
  int st = PSB_OK;
  Cx<T>* A = scratch<T>(c, "dsmag.A", (size_t)12 * fs, &st);
  Cx<T>* B = scratch<T>(c, "dsmag.B", (size_t)12 * fs, &st);
  double* g = reinterpret_cast<double*>(scratch<double>(c, "dsmag.g", (size_t)(N1 + N2 + N3h), &st));
  double* part = reinterpret_cast<double*>(scratch<double>(c, "dsmag.part", kLmBlocks, &st));
  double* cs2 = reinterpret_cast<double*>(scratch<double>(c, "dsmag.cs2", 2, &st));
  if (st != PSB_OK) return st;
  // test filter kL = kc/alpha, alpha = 2 (:1695-1697); a fractional kL is truncated
  const int kl = (int)(c->kc / 2.0);
  if (c->dsmag_kl != kl) {
    std::vector<double> h(N1 + N2 + N3h);
    myfilter_rows(N1, kl, true, h.data());
    myfilter_rows(N2, kl, true, h.data() + N1);
    myfilter_rows(N3h, kl, false, h.data() + N1 + N2);
    PSB_TRY(cuda_ok(c, cudaMemcpy(g, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice), "filter upload"));
    c->dsmag_kl = kl;
  }
  const Cx<T>* Qin = io.Q;
  EpiStore<T, 12> sa{A, fs, N2, N3h}, sb{B, fs, N2, N3h};
  const PhysSmag<T> ss{(T)-0.5};  // -2 (-1/2) |S| S_ij = |S| S_ij
  PSB_TRY(run_ns32<T>(c, Qin, PreStrain<T>{}, ss, sa, ts));
  PSB_TRY(run_ns32<T>(c, Qin, PreStrainFiltered<T>(g, g + N1, g + N1 + N2), ss, sb, ts));
  if (!Qin) return PSB_OK;  // allocation only
  const double d2 = -2.0 * c->Delta * c->Delta;
  {
    LaunchScope ls(c, "dsmag L:M reduction", (double)sizeof(Cx<T>) * 24 * fs);
    dsmag_lm_kernel<T><<<kLmBlocks, 256, 0, c->stream>>>(A, B, g, N1, N2, N3, N3h, d2, part);
  }
  PSB_TRY(launch_ok(c, "dsmag L:M"));
  {
    LaunchScope ls(c, "dsmag Cs^2", 16.0 * kLmBlocks);
    dsmag_cs2_kernel<<<1, 256, 0, c->stream>>>(part, kLmBlocks, cs2);
  }
  PSB_TRY(launch_ok(c, "dsmag Cs^2"));
  EpiNS<T, true> epi{io, ktabs<T>(c->kx, c->ky, c->kz), (T)p->nu, p->rotate, (T)p->Om1, (T)p->Om2,
                     (T)p->Om3, 0, N1 / 2, N2 / 2, N3 / 2};
  const int blocks = (int)std::min<long long>((fs + 255) / 256, 4 * 148);
  {
    LaunchScope ls(c, "dsmag epilogue", (double)sizeof(Cx<T>) * 12 * fs + epi.io_bytes(fs));
    dsmag_epi_kernel<T><<<blocks, 256, 0, c->stream>>>(epi, A, N1, N2, N3h, cs2, c->Delta);
  }
  PSB_TRY(launch_ok(c, "dsmag epilogue"));
  if (cs2_out) {
    double h[3];
    PSB_TRY(cuda_ok(c, cudaMemcpyAsync(h, cs2, sizeof(h), cudaMemcpyDeviceToHost, c->stream), "Cs^2 copy"));
    PSB_TRY(cuda_ok(c, cudaStreamSynchronize(c->stream), "Cs^2 sync"));
    *cs2_out = h[0];
  }
  return PSB_OK;
}

}  // namespace

// ===========================================================================
// dispatch
// ===========================================================================
namespace psbh {

template <typename T>
StepIO<T> make_io(psb_ctx* c, void* Q, void* Q0, void* comp, void* rhs, void* read_out, void* w0, int mode,
                  double dtc) {
  StepIO<T> io{};
  io.Q = reinterpret_cast<Cx<T>*>(Q);
  io.Q0 = reinterpret_cast<Cx<T>*>(Q0);
  io.comp = reinterpret_cast<Cx<T>*>(comp);
  io.rhs_out = reinterpret_cast<Cx<T>*>(rhs);
  io.read_out = reinterpret_cast<Cx<T>*>(read_out);
  io.w0_out = reinterpret_cast<Cx<T>*>(w0);
  io.fstride = (long long)c->N1 * c->N2 * c->N3h;
  io.n2 = c->N2;
  io.n3h = c->N3h;
  io.mode = mode;
  io.dtc = (T)dtc;
  return io;
}

template StepIO<double> make_io<double>(psb_ctx*, void*, void*, void*, void*, void*, void*, int, double);
template StepIO<float> make_io<float>(psb_ctx*, void*, void*, void*, void*, void*, void*, int, double);

int dtau_rhs_d(psb_ctx* c, StepIO<double> io, const psb_params* p, double* tau_out);
int dtau_rhs_f(psb_ctx* c, StepIO<float> io, const psb_params* p, double* tau_out);

template <typename T>
int rhs_dispatch(psb_ctx* c, int closure, StepIO<T> io, const psb_params* p, double* tau_out) {
  const Cx<T>* Qin = io.Q;
  const auto tit = c->tuned.find(closure);
  const psb_tuned* ts = tit == c->tuned.end() ? nullptr : &tit->second;
  switch (closure) {
    case PSB_DNS:
    case PSB_SMAG: {
      const bool smag = closure == PSB_SMAG;
      if (smag) {
        const double csd2 = 0.16 * c->Delta * 0.16 * c->Delta;
        if (!io.w0_out)
          return run_ns32<T>(c, Qin, PreStrain<T>{}, PhysSmag<T>{(T)csd2},
                             EpiSmagStep<T>{io, ktabs<T>(c->kx, c->ky, c->kz), (T)p->nu, p->rotate, (T)p->Om1,
                                            (T)p->Om2, (T)p->Om3},
                             ts);
        EpiNS<T, true> epi{io, ktabs<T>(c->kx, c->ky, c->kz), (T)p->nu, p->rotate, (T)p->Om1, (T)p->Om2,
                           (T)p->Om3, 0, c->N1 / 2, c->N2 / 2, c->N3 / 2};
        return run_ns32<T>(c, Qin, PreStrain<T>{}, PhysSmag<T>{(T)csd2}, epi, ts);
      }
      EpiNS<T, false> epi{io, ktabs<T>(c->kx, c->ky, c->kz), (T)p->nu, p->rotate, (T)p->Om1, (T)p->Om2,
                          (T)p->Om3, 1, c->N1 / 2, c->N2 / 2, c->N3 / 2};
      return run_ns32<T>(c, Qin, PreCopyN<T, 3>{}, PhysProducts<T>{}, epi, ts);
    }
    case PSB_MHD: {
      EpiMHD<T> epi{io, ktabs<T>(c->kx, c->ky, c->kz), c->mx, c->my, c->mz,
                    reinterpret_cast<const Cx<T>*>(p->force), (T)p->nu, (T)(p->eta < 0 ? p->nu : p->eta)};
      return run_mhd<T>(c, Qin, epi);
    }
    case PSB_MHD_TMODEL:
      return run_mhd_tmodel<T>(c, io, p);
    case PSB_TMODEL:
    case PSB_TAU_STATIC: {
      int st = PSB_OK;
      Cx<T>* PLp = scratch<T>(c, "mem.PLp", (size_t)3 * c->N1 * c->N2 * c->N3h, &st);
      if (st != PSB_OK) return st;
      MemCfg m{"memu", nullptr, 0, true, false, 0};
      Cx<T>*B2 = nullptr, *E = nullptr;
      if (Qin) {
        st = cuda_ok(c, cudaMemsetAsync(PLp, 0, sizeof(Cx<T>) * 3 * c->N1 * c->N2 * c->N3h, c->stream), "memset");
        if (st != PSB_OK) return st;
      }
      PSB_TRY(run_pl<T>(c, Qin, p, m, &B2, &E, PLp, nullptr));
      double coef;
      if (closure == PSB_TMODEL) {
        coef = p->Ct * p->t;
      } else {
        const double tau = p->tau_a + p->tau_b * p->t;
        if (tau_out) *tau_out = tau;
        coef = tau > 0.0 ? tau : 0.0;
      }
      EpiPLQL<T> epi{};
      epi.io = io;
      epi.k = ktabs<T>(c->kx, c->ky, c->kz);
      epi.PLp = PLp;
      epi.coef = (T)coef;
      epi.rotate = p->rotate;
      epi.Om1 = (T)p->Om1;
      epi.Om2 = (T)p->Om2;
      epi.Om3 = (T)p->Om3;
      epi.ny1 = c->N1 / 2;
      epi.ny2 = c->N2 / 2;
      epi.ny3 = c->N3 / 2;
      epi.plql_out = nullptr;
      return run_plql<T>(c, m, Qin ? B2 : nullptr, E, epi);
    }
    case PSB_DSMAG:
      return dsmag_rhs<T>(c, io, p, ts, tau_out);
    case PSB_CM1:
      return cm1_rhs<T>(c, io, p);
    case PSB_BUDGETS:
      return budgets_rhs<T>(c, io, p);
    case PSB_FM1:
      return fm1_rhs<T>(c, io, p);
    case PSB_FM2:
      return fm2_rhs<T>(c, io, p);
    case PSB_ORTHO:
      return ortho_rhs<T>(c, io, p, ts);
    case PSB_MPI_DNS:
      return mpi_ns_rhs<T>(c, io, p, false);
    case PSB_MPI_ORTHO:
      return mpi_ns_rhs<T>(c, io, p, true);
    case PSB_TAU_DYNAMIC:
      if constexpr (sizeof(T) == 8)
        return dtau_rhs_d(c, io, p, tau_out);
      else
        return dtau_rhs_f(c, io, p, tau_out);
    case PSB_LEARNED: {
      if (Qin && (!p->mlp_params || !p->mlp_norm))
        return fail(c, PSB_ERR_ARG, "PSB_LEARNED needs mlp_params and mlp_norm");
      if (p->mlp_act != PSB_ACT_GELU && p->mlp_act != PSB_ACT_RELU)
        return fail(c, PSB_ERR_ARG, "PSB_LEARNED: mlp_act must be PSB_ACT_GELU or PSB_ACT_RELU");
      if (!(p->mlp_hidden == 0 || p->mlp_hidden == 64 || (p->mlp_hidden == 32 && p->mlp_act == PSB_ACT_RELU)))
        return fail(c, PSB_ERR_ARG, "PSB_LEARNED: mlp_hidden must be 64 (0), or 32 with PSB_ACT_RELU");
      EpiNS<T, false> epi{io, ktabs<T>(c->kx, c->ky, c->kz), (T)p->nu, p->rotate, (T)p->Om1, (T)p->Om2,
                          (T)p->Om3, 1, c->N1 / 2, c->N2 / 2, c->N3 / 2};
      const double s32 = std::sqrt(std::pow(1.5, 3) * std::sqrt((double)c->N1 * c->N2 * c->N3));
      const float* mp = reinterpret_cast<const float*>(p->mlp_params);
      const float* mn = reinterpret_cast<const float*>(p->mlp_norm);
      const float delta = (float)(p->les_delta > 0 ? p->les_delta : c->Delta);
      // width-32 networks are built with ReLU only
      if (p->mlp_act == PSB_ACT_GELU)
        return run_ns32<T>(c, Qin, PreGradXY<T>{}, PhysLearned<T, kActGelu>{mp, mn, (T)s32, delta}, epi, ts);
      if (p->mlp_hidden == 32)
        return run_ns32<T>(c, Qin, PreGradXY<T>{}, PhysLearned<T, kActRelu, 32>{mp, mn, (T)s32, delta}, epi, ts);
      return run_ns32<T>(c, Qin, PreGradXY<T>{}, PhysLearned<T, kActRelu>{mp, mn, (T)s32, delta}, epi, ts);
    }
    default:
      return fail(c, PSB_ERR_UNSUPPORTED, "unknown closure");
  }
}

int si_step(psb_ctx* c, void* Q, void* H, void* read_out, const psb_params* p) {
  if (c->prec == 64)
    return mpi_si_step<double>(c, reinterpret_cast<Cx<double>*>(Q), reinterpret_cast<Cx<double>*>(H),
                               reinterpret_cast<Cx<double>*>(read_out), p);
  return mpi_si_step<float>(c, reinterpret_cast<Cx<float>*>(Q), reinterpret_cast<Cx<float>*>(H),
                            reinterpret_cast<Cx<float>*>(read_out), p);
}

template int rhs_dispatch<double>(psb_ctx*, int, StepIO<double>, const psb_params*, double*);
template int rhs_dispatch<float>(psb_ctx*, int, StepIO<float>, const psb_params*, double*);

// ---------------------------------------------------------------------------
// Autotuning of a single run's five NS passes (DNS, Smagorinsky, learned).
// Each candidate shape of a pass (column tile or pencils per CTA, and every
// radix order of the default and the fewest-pass schedules) is timed with
// CUDA events inside full RHS evaluations through the single-run kernels, in
// a middle-RK-stage mode on scratch copies of the caller's state (so the
// state is never written).  The default shape is the incumbent: a candidate
// must beat it by 3% and win again in a longer re-timing.
// ---------------------------------------------------------------------------
namespace tuning {

void clear_records(psb_ctx* c) {
  for (auto& r : c->recs) {
    c->ev_free.push_back(r.a);
    c->ev_free.push_back(r.b);
  }
  c->recs.clear();
}

bool plan_is_wide(const FFTPlan& p) {
  for (int s = 0; s < p.npass; ++s)
    if (p.radix[s] > 8 || p.radix[s] == 6) return true;
  return false;
}

// Field counts and limits of the five passes of a tunable closure.
// Fi / Fb: fields after the x / y pass; Fz: z-pass inputs (its smem bound);
// Fy / Gy: lines per column and outer groups of the y-inverse pass
struct TuneDims {
  int Fi, Fb, Fz, Fo, maxppc, defppc, Fy = 1, Gy;
  size_t zextra = 0;
  int Ls[5], Fs[5];
  int zP = 0;  // the register z pass's pencils per CTA and plan (0: none at this length)
  FFTPlan zplan{};
};

template <typename T>
TuneDims tune_dims(psb_ctx* c, int closure, int act, int hidden) {
  TuneDims t;
  if (closure == PSB_DNS) {
    t.Fi = t.Fb = t.Gy = 3, t.Fo = 6, t.maxppc = phys_max_ppc<PhysProducts<T>>::value;
    t.Fz = PhysProducts<T>::F_IN;
    t.defppc = phys_default_ppc<PhysProducts<T>>::value;
  } else if (closure == PSB_SMAG) {
    t.Fi = PreStrain<T>::F_DST, t.Fb = pre_b_fields<PreStrain<T>>::value, t.Fo = 12;
    t.Fy = pre_tile_fields<PreYStrain<T>>();
    t.Gy = pre_ypass<T, PreStrain<T>>::groups * pre_tile_groups<PreYStrain<T>>();
    t.maxppc = phys_max_ppc<PhysSmag<T>>::value;
    t.Fz = PhysSmag<T>::F_IN;
    t.defppc = phys_default_ppc<PhysSmag<T>>::value;
  } else {
    t.Fi = PreGradXY<T>::F_DST, t.Fb = pre_b_fields<PreGradXY<T>>::value, t.Fo = 6;
    t.Fy = PreYGrad<T>::F_DST;
    t.Gy = pre_ypass<T, PreGradXY<T>>::groups;
    t.Fz = PhysLearned<T>::F_IN;
    t.maxppc = phys_max_ppc<PhysLearned<T>>::value;
    t.defppc = phys_default_ppc<PhysLearned<T>>::value;
    t.zextra = (size_t)phys_is_block<PhysLearned<T>>::extra;
  }
  const int M1 = 3 * c->N1 / 2, M2 = 3 * c->N2 / 2, M3 = 3 * c->N3 / 2;
  const long long np = (long long)M1 * M2;
  t.zplan = *plan_for(c, M3);
  if (!c->use_zrr) {
  } else if (closure == PSB_DNS) {
    if (has_reg_z<T, PhysProducts<T>>(M3)) t.zP = reg_z_shape<T, PhysProducts<T>>(M3, np, t.zplan);
  } else if (closure == PSB_SMAG) {
    if (has_reg_z<T, PhysSmag<T>>(M3)) t.zP = reg_z_shape<T, PhysSmag<T>>(M3, np, t.zplan);
  } else if (act == PSB_ACT_RELU) {
    using Ph32 = PhysLearned<T, kActRelu, 32>;
    using Ph64 = PhysLearned<T, kActRelu, 64>;
    if (has_reg_z<T, Ph32>(M3))
      t.zP = hidden == 32 ? reg_z_shape<T, Ph32>(M3, np, t.zplan) : reg_z_shape<T, Ph64>(M3, np, t.zplan);
  }
  const int Ls[5] = {M1, M2, M3, M2, M1};
  const int Fs[5] = {t.Fi, t.Fy, 0, 1, t.Fo};
  for (int k = 0; k < 5; ++k) {
    t.Ls[k] = Ls[k];
    t.Fs[k] = Fs[k];
  }
  return t;
}

// Shared memory of pass k with tile `tile` (columns, or pencils per CTA for the z pass).
template <typename T>
size_t pass_smem(const TuneDims& t, int k, int tile) {
  if (k == 2) return zpass_smem_bytes<T>(std::max(t.Fz, t.Fo), tile, t.Ls[2], t.zextra);
  return (size_t)(t.Ls[k] + 2 * (size_t)t.Ls[k] * t.Fs[k] * tile) * sizeof(Cx<T>);
}

// Untuned shape of axis pass k (x-inverse, y-inverse, y-forward, x-forward).
template <typename T>
void default_pass_shape(psb_ctx* c, const TuneDims& t, int k, psb_pass_shape& sh) {
  if (k == 4) {
    // every tunable closure's epilogue has the same line (x_min_warps)
    sh.reg = x_pass_in_registers<T, EpiNS<T, false>>(t.Ls[4], c->N3 / 2, c->N2);
    default_x_shape<T>(c, t.Ls[4], c->N3 / 2, t.Fs[4], c->N2, sh.reg, sh.tile, sh.plan);
    return;
  }
  const int nouter = k == 0 ? c->N2 : (k == 1 ? t.Gy * t.Ls[0] : t.Fo * t.Ls[0]);
  const bool reg = k != 2 && k != 4;
  default_axis_shape<T>(c, t.Ls[k], c->N3 / 2, t.Fs[k], nouter, reg, sh.tile, sh.plan);
  sh.reg = reg && has_reg_axis(t.Ls[k]);
}

template <typename T>
int tune_rhs(psb_ctx* c, int closure, const void* state, const psb_params* p) {
  const int N1 = c->N1, N2 = c->N2, N3 = c->N3, N3h = c->N3h;
  const int M1 = 3 * N1 / 2, M2 = 3 * N2 / 2, M3 = 3 * N3 / 2, Kz = N3 / 2;
  const TuneDims td = tune_dims<T>(c, closure, p->mlp_act, p->mlp_hidden);
  const int Fz = td.Fz, Fo = td.Fo, maxppc = td.maxppc, defppc = td.defppc;
  const size_t zextra = td.zextra;
  const size_t esz = sizeof(Cx<T>);
  const size_t n = (size_t)3 * N1 * N2 * N3h;
  int st = PSB_OK;
  Cx<T>* q = scratch<T>(c, "tune.Q", n, &st);
  Cx<T>* q0 = scratch<T>(c, "tune.Q0", n, &st);
  Cx<T>* cp = c->prec == 32 ? scratch<T>(c, "tune.C", n, &st) : nullptr;
  if (st != PSB_OK) return st;
  PSB_TRY(cuda_ok(c, cudaMemcpyAsync(q, state, n * esz, cudaMemcpyDeviceToDevice, c->stream), "tune copy"));
  PSB_TRY(cuda_ok(c, cudaMemcpyAsync(q0, state, n * esz, cudaMemcpyDeviceToDevice, c->stream), "tune copy"));
  if (cp) PSB_TRY(cuda_ok(c, cudaMemsetAsync(cp, 0, n * esz, c->stream), "tune memset"));
  const StepIO<T> io = make_io<T>(c, q, q0, cp, nullptr, nullptr, nullptr, kStageMid, p->dt / 3.0);
  const int FMAX = std::max(Fz, Fo);
  auto zsmem = [&](int P) { return zpass_smem_bytes<T>(FMAX, P, M3, zextra); };
  int P = defppc;
  while (P > 1 && zsmem(P) > kSmemBudget) P /= 2;
  while (P > 1 && ((long long)M1 * M2 + P - 1) / P < 2 * 148) P /= 2;
  psb_tuned t;
  const int* Ls = td.Ls;
  const int* Fs = td.Fs;
  for (int k : {0, 1, 3, 4}) default_pass_shape<T>(c, td, k, t.pass[k]);
  t.pass[2].tile = td.zP ? td.zP : P;
  t.pass[2].plan = td.zplan;
  t.pass[2].reg = td.zP > 0;
  c->tuned[closure] = t;
  static const char* names[5] = {"x-inverse", "y-inverse", "z-fused", "y-forward", "x-forward+epilogue"};
  const int timing_was = c->timing;
  clear_records(c);
  c->timing = 1;
  auto time_pass = [&](int k, int reps, float* ms) -> int {
    clear_records(c);
    for (int r = 0; r < reps + 1; ++r) PSB_TRY(rhs_dispatch<T>(c, closure, io, p, nullptr));
    PSB_TRY(cuda_ok(c, cudaStreamSynchronize(c->stream), "tune sync"));
    // the fastest of the timed launches: a launch slowed by something outside
    // the candidate (a clock step, another stream) does not decide the choice
    float best = 1e30f;
    int seen = 0;
    for (const auto& rec : c->recs) {
      if (rec.name != names[k]) continue;
      if (seen++ == 0) continue;  // the first evaluation warms up
      float e = 0.f;
      PSB_TRY(cuda_ok(c, cudaEventElapsedTime(&e, rec.a, rec.b), "tune elapsed"));
      best = std::min(best, e);
    }
    *ms = best;
    return PSB_OK;
  };
  int status = PSB_OK;
  for (int k = 0; k < 5 && status == PSB_OK; ++k) {
    psb_pass_shape& cur = c->tuned[closure].pass[k];
    const psb_pass_shape inc = cur;
    // the register z pass is chosen by psb_ctx_set_zrr, not by a shape
    if (k == 2 && inc.reg) continue;
    float base = 0.f;
    if ((status = time_pass(k, 6, &base)) != PSB_OK) break;
    std::vector<int> tiles;
    if (k == 2) {
      for (int pp : {1, 2, 4, 8})
        if (pp <= maxppc && zsmem(pp) <= kSmemBudget) tiles.push_back(pp);
    } else {
      for (int ct : {2, 4, 8, 16, 32})
        if (ct <= std::max(2, 2 * Kz) && (size_t)(Ls[k] + 2 * Ls[k] * Fs[k] * ct) * esz <= kSmemBudget)
          tiles.push_back(ct);
    }
    psb_pass_shape best = inc;
    float bms = 0.97f * base;
    if (k == 4 && !inc.reg && has_reg_x(Ls[4])) {  // the register pass where the default is the staged one
      default_x_shape<T>(c, Ls[4], Kz, Fs[4], N2, true, cur.tile, cur.plan);
      cur.reg = true;
      float ms = 0.f;
      if ((status = time_pass(k, 6, &ms)) != PSB_OK) break;
      if (ms < bms) {
        bms = ms;
        best = cur;
      }
    }
    for (int tl : tiles) {
      for (const FFTPlan& q2 : radix_orders(*plan_for(c, Ls[k]))) {
        cur.tile = tl;
        cur.plan = q2;
        cur.wide = plan_is_wide(q2);
        cur.reg = false;
        float ms = 0.f;
        if ((status = time_pass(k, 6, &ms)) != PSB_OK) break;
        if (ms < bms) {
          bms = ms;
          best = cur;
        }
      }
      if (status != PSB_OK) break;
    }
    if (status != PSB_OK) break;
    cur = best;
    if (best.reg != inc.reg || best.tile != inc.tile || best.plan.npass != inc.plan.npass ||
        !std::equal(best.plan.radix, best.plan.radix + best.plan.npass, inc.plan.radix)) {
      float again = 0.f, def = 0.f;
      if ((status = time_pass(k, 10, &again)) != PSB_OK) break;
      cur = inc;
      if ((status = time_pass(k, 10, &def)) != PSB_OK) break;
      cur = again < 0.98f * def ? best : inc;
    }
  }
  clear_records(c);
  c->timing = timing_was;
  if (status != PSB_OK) c->tuned.erase(closure);
  return status;
}

// A caller-given launch shape for pass k of `closure` (a saved autotuner
// result, or a shape a test wants to exercise): checked against the pass's
// transform length, the radices the kernels have and the shared-memory budget.
bool staged_radix(int r) { return r == 2 || r == 3 || r == 4 || r == 6 || r == 8 || r == 12 || r == 16; }

template <typename T>
int set_shape(psb_ctx* c, int closure, int k, int tile, const int* radices, int nrad) {
  const TuneDims td = tune_dims<T>(c, closure, PSB_ACT_RELU, 32);
  const int L = td.Ls[k];
  if (nrad < 1 || nrad > kMaxPasses) return fail(c, PSB_ERR_ARG, "psb_set_tuned_shape: 1..12 radices");
  long long prod = 1;
  bool wide = false;
  FFTPlan q = *plan_for(c, L);
  q.npass = nrad;
  // the register pass is named by its radices and its tile, or by its radices alone
  // where the staged passes do not have them
  FFTPlan rp = q;
  bool reg_shape = false;
  if (k == 2) {
    reg_shape = td.zP > 0 && nrad == 3 && std::equal(radices, radices + 3, td.zplan.radix) && tile >= 1 &&
                tile <= 128;
  } else if (k == 4 ? reg_x_plan(L, rp) : reg_axis_plan(L, rp)) {
    reg_shape = nrad == rp.npass && std::equal(radices, radices + nrad, rp.radix) &&
                (tile == (k == 4 ? xreg_cols<T>() : reg_cols<T>()) || !std::all_of(radices, radices + nrad, staged_radix));
  }
  for (int s = 0; s < nrad; ++s) {
    const int r = radices[s];
    if (reg_shape) {
      q.radix[s] = r;
      prod *= r;
      continue;
    }
    if (!staged_radix(r))
      return fail(c, PSB_ERR_ARG, "psb_set_tuned_shape: radices must be 2, 3, 4, 6, 8, 12 or 16");
    wide = wide || r > 8 || r == 6;
    prod *= r;
    q.radix[s] = r;
  }
  for (int s = nrad; s < kMaxPasses; ++s) q.radix[s] = 0;
  if (prod != L)
    return fail(c, PSB_ERR_SHAPE, "psb_set_tuned_shape: the radices multiply to " + std::to_string(prod) +
                                      ", the pass transforms " + std::to_string(L) + " points");
  const int tmax = k == 2 ? td.maxppc : 32;
  if (!(k == 2 && reg_shape) && (tile < 1 || tile > tmax || (tile & (tile - 1))))
    return fail(c, PSB_ERR_ARG, "psb_set_tuned_shape: tile must be a power of two <= " + std::to_string(tmax));
  if (!reg_shape && pass_smem<T>(td, k, tile) > kSmemBudget)
    return fail(c, PSB_ERR_SHAPE, "psb_set_tuned_shape: tile needs more shared memory than the budget");
  auto it = c->tuned.find(closure);
  if (it == c->tuned.end()) {
    // start from the default shapes of every pass
    psb_tuned t;
    int P = td.defppc;
    while (P > 1 && pass_smem<T>(td, 2, P) > kSmemBudget) P /= 2;
    while (P > 1 && ((long long)td.Ls[0] * td.Ls[1] + P - 1) / P < 2 * 148) P /= 2;
    for (int j : {0, 1, 3, 4}) default_pass_shape<T>(c, td, j, t.pass[j]);
    t.pass[2].tile = td.zP ? td.zP : P;
    t.pass[2].plan = td.zplan;
    t.pass[2].reg = td.zP > 0;
    it = c->tuned.emplace(closure, t).first;
  }
  psb_pass_shape& sh = it->second.pass[k];
  sh.tile = tile;
  sh.plan = q;
  sh.wide = wide;
  sh.reg = reg_shape;
  return PSB_OK;
}

}  // namespace tuning

// SGS of a filtered DNS field
template <typename T>
int sgs_dns_run(psb_ctx* c, const void* fields, void* w0, void* tau6) {
  EpiSGSDNS<T> epi{ktabs<T>(c->kx, c->ky, c->kz), c->gx, c->gy, c->gz, reinterpret_cast<Cx<T>*>(w0),
                   reinterpret_cast<Cx<T>*>(tau6), (long long)c->N1 * c->N2 * c->N3h, c->N2, c->N3h};
  PreFiltered<T> pre{c->gx, c->gy, c->gz};
  return run_ns32<T>(c, reinterpret_cast<const Cx<T>*>(fields), pre, PhysSGSDNS<T>{}, epi);
}
template int sgs_dns_run<double>(psb_ctx*, const void*, void*, void*);
template int sgs_dns_run<float>(psb_ctx*, const void*, void*, void*);

// The six dealiased product spectra (uuhat.. of src/RHSfunctions.py:18-23).
template <typename T>
int products_run(psb_ctx* c, const void* fields, void* out6) {
  EpiStore<T, 6> epi{reinterpret_cast<Cx<T>*>(out6), (long long)c->N1 * c->N2 * c->N3h, c->N2, c->N3h};
  return run_ns32<T>(c, reinterpret_cast<const Cx<T>*>(fields), PreCopyN<T, 3>{}, PhysProducts<T>{}, epi);
}
template int products_run<double>(psb_ctx*, const void*, void*);
template int products_run<float>(psb_ctx*, const void*, void*);

// the six products of Gf u (the sharp-cutoff filtered field; transfer of the resolved scales)
template <typename T>
int products_filtered_run(psb_ctx* c, const void* fields, void* out6) {
  EpiStore<T, 6> epi{reinterpret_cast<Cx<T>*>(out6), (long long)c->N1 * c->N2 * c->N3h, c->N2, c->N3h};
  return run_ns32<T>(c, reinterpret_cast<const Cx<T>*>(fields), PreMask3<T>{c->gx, c->gy, c->gz},
                     PhysProducts<T>{}, epi);
}
template int products_filtered_run<double>(psb_ctx*, const void*, void*);
template int products_filtered_run<float>(psb_ctx*, const void*, void*);

// exported for the dynamic tau-model translation unit
template <typename T>
int mem_stage_pl(psb_ctx* c, const Cx<T>* Qin, const psb_params* p, const char* tag, const double* filt, int kfp,
                 Cx<T>* PLp, Cx<T>* Lbox, int kfb, Cx<T>** B2, Cx<T>** E) {
  MemCfg m{tag, filt, kfp, PLp != nullptr, Lbox != nullptr, kfb};
  return run_pl<T>(c, Qin, p, m, B2, E, PLp, Lbox);
}
template <typename T>
int mem_stage_plql(psb_ctx* c, Cx<T>* B2, Cx<T>* E, EpiPLQL<T> epi) {
  MemCfg m{"", nullptr, 0, false, false, 0};
  return run_plql<T>(c, m, B2, E, epi);
}
template int mem_stage_pl<double>(psb_ctx*, const Cx<double>*, const psb_params*, const char*, const double*, int,
                                  Cx<double>*, Cx<double>*, int, Cx<double>**, Cx<double>**);
template int mem_stage_pl<float>(psb_ctx*, const Cx<float>*, const psb_params*, const char*, const double*, int,
                                 Cx<float>*, Cx<float>*, int, Cx<float>**, Cx<float>**);
template int mem_stage_plql<double>(psb_ctx*, Cx<double>*, Cx<double>*, EpiPLQL<double>);
template int mem_stage_plql<float>(psb_ctx*, Cx<float>*, Cx<float>*, EpiPLQL<float>);

}  // namespace psbh

extern "C" int psb_autotune(psb_ctx* c, int closure, void* state, const psb_params* p) {
  if (!c) return PSB_ERR_ARG;
  if (!state || !p) return fail(c, PSB_ERR_ARG, "psb_autotune: null argument");
  if (closure != PSB_DNS && closure != PSB_SMAG && closure != PSB_LEARNED)
    return fail(c, PSB_ERR_UNSUPPORTED, "psb_autotune: closure not tunable (DNS, SMAG, LEARNED are)");
  if (closure == PSB_LEARNED && (!p->mlp_params || !p->mlp_norm))
    return fail(c, PSB_ERR_ARG, "psb_autotune: PSB_LEARNED needs mlp_params and mlp_norm");
  if (closure == PSB_LEARNED && p->mlp_act != PSB_ACT_GELU && p->mlp_act != PSB_ACT_RELU)
    return fail(c, PSB_ERR_ARG, "psb_autotune: mlp_act must be PSB_ACT_GELU or PSB_ACT_RELU");
  if (closure == PSB_LEARNED &&
      !(p->mlp_hidden == 0 || p->mlp_hidden == 64 || (p->mlp_hidden == 32 && p->mlp_act == PSB_ACT_RELU)))
    return fail(c, PSB_ERR_ARG, "psb_autotune: mlp_hidden must be 64 (0), or 32 with PSB_ACT_RELU");
  PSB_TRY(cuda_ok(c, cudaSetDevice(c->dev), "cudaSetDevice"));
  return c->prec == 64 ? psbh::tuning::tune_rhs<double>(c, closure, state, p)
                        : psbh::tuning::tune_rhs<float>(c, closure, state, p);
}

extern "C" int psb_set_tuned_shape(psb_ctx* c, int closure, int pass, int tile, const int* radices, int nrad) {
  if (!c) return PSB_ERR_ARG;
  if (closure != PSB_DNS && closure != PSB_SMAG && closure != PSB_LEARNED)
    return fail(c, PSB_ERR_UNSUPPORTED, "psb_set_tuned_shape: closure not tunable (DNS, SMAG, LEARNED are)");
  if (pass < 0 || pass > 4 || !radices) return fail(c, PSB_ERR_ARG, "psb_set_tuned_shape: bad argument");
  return c->prec == 64 ? psbh::tuning::set_shape<double>(c, closure, pass, tile, radices, nrad)
                        : psbh::tuning::set_shape<float>(c, closure, pass, tile, radices, nrad);
}

