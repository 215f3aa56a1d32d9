// Pointwise physics of the right-hand sides: spectral expanders run on load by
// the x-inverse pass, physical-space products run inside the z-pass, spectral
// epilogues (projection, viscosity, closure, Coriolis, RK stage) run after the
// last forward pass.  Every formula cites the reference line it restates.
#pragma once
#include "psb_passes.cuh"

namespace psb {

// ---- precision helpers ---------------------------------------------------
// FP64 keeps the reference's ksqr = k.k + 1e-50 and ksqr_i = 1/ksqr
// (PySpectral/src/Classes.py:576-577).  In FP32 1e-50 flushes to zero, so the
// k=0 mode uses ksqr_i = 0; every term it multiplies vanishes there anyway.
template <typename T>
__device__ __forceinline__ void ksq_pair(T k1, T k2, T k3, T& ksq, T& ksqi) {
  if constexpr (sizeof(T) == 8) {
    ksq = k1 * k1 + k2 * k2 + k3 * k3 + 1.0e-50;
    ksqi = 1.0 / ksq;
  } else {
    ksq = k1 * k1 + k2 * k2 + k3 * k3;
    ksqi = ksq > (T)0 ? (T)1 / ksq : (T)0;
  }
}

// -i*k*X and i*k*X
template <typename T>
__device__ __forceinline__ Cx<T> mik(T k, Cx<T> X) { return mk<T>(k * X.y, -k * X.x); }
template <typename T>
__device__ __forceinline__ Cx<T> pik(T k, Cx<T> X) { return mk<T>(-k * X.y, k * X.x); }

// ---- RK stage bookkeeping --------------------------------------------------
enum StageMode : int { kRHS = 0, kStage1 = 1, kStageMid = 2, kStageLast = 3 };

template <typename T>
struct StepIO {
  Cx<T>* Q;         // state (read; updated in RK modes)
  Cx<T>* Q0;        // step start state (written in stage 1)
  Cx<T>* comp;      // Kahan compensation (FP32 runs) or null
  Cx<T>* rhs_out;   // RHS output (kRHS) or null
  Cx<T>* read_out;  // state as read by this RHS (the reference's main.uhat) or null
  Cx<T>* w0_out;    // closure force (main.w0_*) or null
  long long fstride;
  int n2, n3h;
  int mode;
  T dtc;  // dt * rk4const[i]
  __device__ __forceinline__ long long sidx(int i1, int i2, int i3) const {
    return ((long long)i1 * n2 + i2) * n3h + i3;
  }
  // compulsory state traffic over npts points and nf fields
  __host__ double bytes(long long npts, int nf) const {
    double n = 1.0;  // read Q
    if (mode == kRHS) n += 1.0;
    else n += 2.0 + (comp ? (mode == kStageLast ? 2.0 : 1.0) : 0.0);
    if (read_out) n += 1.0;
    double b = n * (double)sizeof(Cx<T>) * npts * nf;
    if (w0_out) b += (double)sizeof(Cx<T>) * npts * 3;
    return b;
  }
  // What finish() reads of one mode and field, so that a caller can issue the
  // loads of several modes before the first store.
  struct Old {
    Cx<T> base, c;
  };
  // q: the state at this mode, when the caller has read it (stage 1 starts from it)
  __device__ __forceinline__ Old fetch(long long s, int f, Cx<T> q) const {
    const long long e = f * fstride + s;
    Old o;
    o.base = q;
    o.c = mk<T>(0, 0);
    if (mode == kStageMid || mode == kStageLast) o.base = Q0[e];
    if (mode != kRHS && comp != nullptr) o.c = comp[e];
    return o;
  }
  // Q = Q0 + dt*c*RHS  (PySpectral/src/PySpec_3d.py:104), Kahan-compensated when comp != null.
  __device__ __forceinline__ void finish(long long s, int f, Cx<T> R, const Old& o) const {
    const long long e = f * fstride + s;
    if (mode == kRHS) {
      rhs_out[e] = R;
      return;
    }
    if (mode == kStage1) Q0[e] = o.base;
    const Cx<T> inc = dtc * R;
    if (comp == nullptr) {
      Q[e] = o.base + inc;
    } else {
      const Cx<T> y = inc - o.c;
      const Cx<T> t = o.base + y;
      if (mode == kStageLast) comp[e] = (t - o.base) - y;
      Q[e] = t;
    }
  }
  __device__ __forceinline__ void finish(long long s, int f, Cx<T> R) const {
    finish(s, f, R, fetch(s, f, mode == kStage1 ? Q[f * fstride + s] : mk<T>(0, 0)));
  }
};

// The state of NF fields at a mode and what the RK stage needs beside it.
template <typename T, int NF>
struct StateIn {
  Cx<T> q[NF];
  typename StepIO<T>::Old o[NF];
  __device__ __forceinline__ void load(const StepIO<T>& io, long long s) {
#pragma unroll
    for (int f = 0; f < NF; ++f) q[f] = io.Q[f * io.fstride + s];
#pragma unroll
    for (int f = 0; f < NF; ++f) o[f] = io.fetch(s, f, q[f]);
  }
};

// field table of a pass that copies fields 0..nf-1, each times m1[row] m2[outer] m3[col] when given
template <typename T>
__host__ inline FieldTab<T> copy_fields(int nf, const double* m1 = nullptr, const double* m2 = nullptr,
                                        const double* m3 = nullptr) {
  FieldTab<T> t;
  t.nf = nf;
  for (int f = 0; f < nf; ++f) t.sa[f] = (unsigned char)f;
  t.m1 = m1;
  t.m2 = m2;
  t.m3 = m3;
  return t;
}

// ---- 3/2-padded Navier-Stokes: DNS and Smagorinsky --------------------------
template <typename T, int F>
struct PreCopyN {
  static constexpr int F_SRC = F, F_DST = F;
  __device__ void operator()(int, int, int, const AxisArgs<T>&, const Cx<T>* s, Cx<T>* d) const {
#pragma unroll
    for (int f = 0; f < F; ++f) d[f] = s[f];
  }
  __host__ FieldTab<T> fields() const { return copy_fields<T>(F); }
};

// The strain S_ij = (i/2)(k_j u_i + k_i u_j) (PySpectral/src/RHSfunctions.py:174-179)
// is formed as late as its derivatives allow, so that the passes carry fewer
// fields than the nine the z pass needs: the x pass u and i k1 u (6), the y pass
// (u, v, w, S11, S22, S12, dw/dx, dw/dy) (8), and the z pass completes
// S33 = i k3 w, S13 = (i k3 u + dw/dx)/2 and S23 = (i k3 v + dw/dy)/2 on load.
template <typename T>
struct PreYStrain {
  static constexpr int F_SRC = 6, F_DST = 8, GROUPS = 1, IN_FIELDS = 1, OUT_FIELDS = 1;
  // the staged pass takes one field a CTA; with the eight in one tile its rows were one
  // column wide (324 x 324 x 64, 486 points: FP64 2.24 ms against 3.17, FP32 1.28
  // against 1.41; 768 points FP64, 48 x 512 x 48, is the exception, 637 us against 549)
  static constexpr bool SPLIT = true;
  // stored fields u, v, w, i k1 u, i k1 v, i k1 w; field g from sa(g) (and sb(g))
  __host__ __device__ static constexpr int sa(int g) {
    return g < 4 ? g : (g == 4 ? 1 : (g == 5 ? 0 : (g == 6 ? 5 : 2)));
  }
  __host__ __device__ static constexpr int sb(int) { return 4; }
  __host__ __device__ static constexpr FieldKind kind(int g) {
    return g < 4 || g == 6 ? kCopy : (g == 5 ? kIkMean : kIkRow);
  }
  __device__ __forceinline__ static Cx<T> split(FieldKind kind, T k, Cx<T> a, Cx<T> b) {
    if (kind == kCopy) return a;
    return kind == kIkRow ? pik(k, a) : (T)0.5 * (pik(k, a) + b);
  }
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t;
    t.nf = 8;
    for (int g = 0; g < 8; ++g) {
      t.sa[g] = (unsigned char)sa(g);
      t.sb[g] = (unsigned char)sb(g);
      t.kind[g] = kind(g);
    }
    return t;
  }
};
template <typename T>
struct PreStrain {
  static constexpr int F_SRC = 3, F_DST = 6, F_B = 8, Z_DERIVED = 1;
  using YPass = PreYStrain<T>;
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t;
    t.nf = 6;
    for (int g = 0; g < 6; ++g) {
      t.sa[g] = (unsigned char)(g % 3);
      t.kind[g] = g < 3 ? kCopy : kIkRow;
    }
    return t;
  }
  __device__ void operator()(int i, int, int, const AxisArgs<T>& a, const Cx<T>* s, Cx<T>* d) const {
    const T k1 = (T)a.k_row[i];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      d[f] = s[f];
      d[3 + f] = pik(k1, s[f]);
    }
  }
  // z-pass inputs u, v, w, S11, S22, S33, S12, S13, S23
  __host__ static void zsrc(int f, int& src, bool& der) {
    const int s[9] = {0, 1, 2, 3, 4, 2, 5, 0, 1};
    src = s[f];
    der = f == 5 || f >= 7;
  }
  __host__ static int zsrc2(int f) { return f < 7 ? -1 : f - 1; }
};

// u_i u_j in physical space (PySpectral/src/RHSfunctions.py:18-23)
template <typename T>
struct PhysProducts {
  static constexpr int F_IN = 3, F_OUT = 6;
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
    const T u = in[0], v = in[1], w = in[2];
    out[0] = u * u;
    out[1] = v * v;
    out[2] = w * w;
    out[3] = u * v;
    out[4] = u * w;
    out[5] = v * w;
  }
};

// Products plus the Smagorinsky stress tau_ij = -2 (Cs Delta)^2 |S| S_ij
// (PySpectral/src/RHSfunctions.py:195-212, Cs = 0.16 at :197).
template <typename T>
struct PhysSmag {
  static constexpr int F_IN = 9, F_OUT = 12;
  static constexpr bool IN2 = true;  // S13 and S23 (PreStrain::zsrc2)
  T csd2;  // 0.16*Delta*0.16*Delta
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
    const T u = in[0], v = in[1], w = in[2];
    out[0] = u * u;
    out[1] = v * v;
    out[2] = w * w;
    out[3] = u * v;
    out[4] = u * w;
    out[5] = v * w;
    const T S11 = in[3], S22 = in[4], S33 = in[5], S12 = in[6], S13 = in[7], S23 = in[8];
    const T sm = sqrt((T)2 * (S11 * S11 + S22 * S22 + S33 * S33 + (T)2 * S12 * S12 + (T)2 * S13 * S13 +
                              (T)2 * S23 * S23));
    const T m2nut = (T)-2 * (csd2 * fabs(sm));
    out[6] = m2nut * S11;
    out[7] = m2nut * S22;
    out[8] = m2nut * S33;
    out[9] = m2nut * S12;
    out[10] = m2nut * S13;
    out[11] = m2nut * S23;
  }
};

template <typename T>
struct KTabs {
  const double *k1, *k2, *k3;
};

// Spectral epilogues in two halves.  acc(f, k1, k2, k3, v, D) adds product
// spectrum f to NACC accumulators D[m][r] of R modes that differ in k1 only;
// ld(i1, i2, i3) reads what one mode needs beside its products, and fin(i1, i2,
// i3, D, in) forms the mode's right-hand side from its NACC sums and stores it
// (apart, so that the loads of several modes are in flight together).  The right-hand sides are linear in the products, so a thread
// needs the sums (the divergence k_j P_ij, and what else a closure contracts)
// and not the products: the register x pass (psb_xreg.cuh) takes the fields one
// after another.  operator() is both for one mode with its F_IN products.
template <int R, typename T>
__device__ __forceinline__ void acc_row(T k, const Cx<T>* v, Cx<T>* D) {
#pragma unroll
  for (int r = 0; r < R; ++r) D[r] = mk<T>(D[r].x + k * v[r].x, D[r].y + k * v[r].y);
}
template <int R, typename T>
__device__ __forceinline__ void acc_row(const T* k, const Cx<T>* v, Cx<T>* D) {
#pragma unroll
  for (int r = 0; r < R; ++r) D[r] = mk<T>(D[r].x + k[r] * v[r].x, D[r].y + k[r] * v[r].y);
}
// D_i += k_j P_ij for symmetric product f of 11, 22, 33, 12, 13, 23
template <int R, typename T>
__device__ __forceinline__ void acc_sym(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*D)[R]) {
  switch (f) {
    case 0:
      acc_row<R>(k1, v, D[0]);
      break;
    case 1:
      acc_row<R>(k2, v, D[1]);
      break;
    case 2:
      acc_row<R>(k3, v, D[2]);
      break;
    case 3:
      acc_row<R>(k2, v, D[0]);
      acc_row<R>(k1, v, D[1]);
      break;
    case 4:
      acc_row<R>(k3, v, D[0]);
      acc_row<R>(k1, v, D[2]);
      break;
    default:
      acc_row<R>(k3, v, D[1]);
      acc_row<R>(k2, v, D[2]);
      break;
  }
}
// both halves for one mode
template <typename T, class Epi>
__device__ __forceinline__ void epi_point(const Epi& e, int i1, int i2, int i3, const Cx<T>* P) {
  const KTabs<T> kt = e.ktabs();
  const T k1 = (T)kt.k1[i1], k2 = (T)kt.k2[i2], k3 = (T)kt.k3[i3];
  Cx<T> D[Epi::NACC][1];
#pragma unroll
  for (int m = 0; m < Epi::NACC; ++m) D[m][0] = mk<T>(0, 0);
#pragma unroll
  for (int f = 0; f < Epi::F_IN; ++f) e.template acc<1>(f, &k1, k2, k3, P + f, D);
  e.fin(i1, i2, i3, &D[0][0], e.ld(i1, i2, i3));
}

// DNS / Smagorinsky epilogue (PySpectral/src/RHSfunctions.py:29-50, :164-232).
// Sums: k_j (u_i u_j)^, and k_j tau_ij^ for Smagorinsky with the closure force kept.
template <typename T, bool SMAG>
struct EpiNS {
  static constexpr int F_IN = SMAG ? 12 : 6, NACC = SMAG ? 6 : 3;
  __host__ double io_bytes(long long npts) const { return io.bytes(npts, 3); }
  StepIO<T> io;
  KTabs<T> k;
  T nu;
  int rotate;
  T Om1, Om2, Om3;
  int zero_nyq;  // unpad(pad(uhat)) on read (:10-12); absent in SMAG
  int ny1, ny2, ny3;
  __device__ __forceinline__ KTabs<T> ktabs() const { return k; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*D)[R]) const {
    if constexpr (SMAG) {
      if (f >= 6) {
        acc_sym<R>(f - 6, k1, k2, k3, v, D + 3);
        return;
      }
    }
    acc_sym<R>(f, k1, k2, k3, v, D);
  }
  using In = StateIn<T, 3>;
  __device__ __forceinline__ In ld(int i1, int i2, int i3) const {
    In in;
    in.load(io, io.sidx(i1, i2, i3));
    return in;
  }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* D, const In& in) const {
    const long long s = io.sidx(i1, i2, i3);
    Cx<T> u[3] = {in.q[0], in.q[1], in.q[2]};
    if (zero_nyq && (i1 == ny1 || i2 == ny2 || i3 == ny3)) u[0] = u[1] = u[2] = mk<T>(0, 0);
    const T kv[3] = {(T)k.k1[i1], (T)k.k2[i2], (T)k.k3[i3]};
    T ksq, ksqi;
    ksq_pair(kv[0], kv[1], kv[2], ksq, ksqi);
    Cx<T> ph = (-ksqi) * (kv[0] * D[0] + kv[1] * D[1] + kv[2] * D[2]);
    Cx<T> c[3];
    if (rotate) {
      c[0] = Om3 * u[1] - Om2 * u[2];
      c[1] = Om1 * u[2] - Om3 * u[0];
      c[2] = Om2 * u[0] - Om1 * u[1];
      // phat -= 2 ksqr_i 1j (k . (u x Om)) (:33-36)
      ph = ph - ((T)2 * ksqi) * mul_i(kv[0] * c[0] + kv[1] * c[1] + kv[2] * c[2]);
    }
    // projected SGS divergence (:215-222); note 1j*k_i*(1j*ksqr_i*(kk:tau))
    Cx<T> kk = mk<T>(0, 0);
    if constexpr (SMAG) kk = ksqi * (kv[0] * D[3] + kv[1] * D[4] + kv[2] * D[5]);
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      Cx<T> r = mul_mi(D[m]) + mik(kv[m], ph) - (nu * ksq) * u[m];
      if constexpr (SMAG) {
        const Cx<T> w0 = mul_mi(D[3 + m]) - kv[m] * kk;
        r = r + w0;
        if (io.w0_out) io.w0_out[m * io.fstride + s] = w0;
      }
      if (rotate) r = r + (T)2 * c[m];  // + 2 u x Om (:47-50)
      if (io.read_out) io.read_out[m * io.fstride + s] = u[m];
      io.finish(s, m, r, in.o[m]);
    }
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
};

// The Smagorinsky epilogue when the closure force itself is not asked for (RK
// stages).  The divergence is linear, so u_i u_j and tau_ij share three sums
// k_j (u_i u_j + tau_ij)^; the projections differ (1j*ksqr_i against ksqr_i),
// which needs the scalar kk:tau^ as well.  With C = uu + tau and s = ksqr_i kk:tau,
//   -1j k_j uu_ij - 1j k_i phat + w0_i = -1j (k_j C_ij - k_i ksqr_i kk:C) - (1 + 1j) k_i s.
template <typename T>
struct EpiSmagStep {
  static constexpr int F_IN = 12, NACC = 4;
  __host__ double io_bytes(long long npts) const { return io.bytes(npts, 3); }
  StepIO<T> io;
  KTabs<T> k;
  T nu;
  int rotate;
  T Om1, Om2, Om3;
  __device__ __forceinline__ KTabs<T> ktabs() const { return k; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*D)[R]) const {
    if (f < 6) {
      acc_sym<R>(f, k1, k2, k3, v, D);
      return;
    }
    acc_sym<R>(f - 6, k1, k2, k3, v, D);
    T kk[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      kk[r] = f == 6 ? k1[r] * k1[r]
                     : (f == 7 ? k2 * k2
                               : (f == 8 ? k3 * k3
                                         : (f == 9 ? (T)2 * k1[r] * k2 : (f == 10 ? (T)2 * k1[r] * k3 : (T)2 * k2 * k3))));
    acc_row<R>(kk, v, D[3]);
  }
  using In = StateIn<T, 3>;
  __device__ __forceinline__ In ld(int i1, int i2, int i3) const {
    In in;
    in.load(io, io.sidx(i1, i2, i3));
    return in;
  }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* D, const In& in) const {
    const long long s = io.sidx(i1, i2, i3);
    const Cx<T> u[3] = {in.q[0], in.q[1], in.q[2]};
    const T kv[3] = {(T)k.k1[i1], (T)k.k2[i2], (T)k.k3[i3]};
    T ksq, ksqi;
    ksq_pair(kv[0], kv[1], kv[2], ksq, ksqi);
    Cx<T> ph = (-ksqi) * (kv[0] * D[0] + kv[1] * D[1] + kv[2] * D[2]);
    Cx<T> c[3];
    if (rotate) {
      c[0] = Om3 * u[1] - Om2 * u[2];
      c[1] = Om1 * u[2] - Om3 * u[0];
      c[2] = Om2 * u[0] - Om1 * u[1];
      ph = ph - ((T)2 * ksqi) * mul_i(kv[0] * c[0] + kv[1] * c[1] + kv[2] * c[2]);
    }
    const Cx<T> t = mk<T>(ksqi * (D[3].x - D[3].y), ksqi * (D[3].x + D[3].y));  // (1 + 1j) s
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      Cx<T> r = mul_mi(D[m]) + mik(kv[m], ph) - kv[m] * t - (nu * ksq) * u[m];
      if (rotate) r = r + (T)2 * c[m];
      if (io.read_out) io.read_out[m * io.fstride + s] = u[m];
      io.finish(s, m, r, in.o[m]);
    }
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
};

// ---- MHD (2/3 rule, unpadded), PySpectral/src_MPI/RHSfunctions.py:95-175 ------
template <typename T>
struct PreMask6 {
  static constexpr int F_SRC = 6, F_DST = 6;
  const double *m1, *m2, *m3;
  __device__ void operator()(int i, int o, int c, const AxisArgs<T>&, const Cx<T>* s, Cx<T>* d) const {
    const T m = (T)(m1[i] * m2[o] * m3[c]);
#pragma unroll
    for (int f = 0; f < 6; ++f) d[f] = m * s[f];
  }
  __host__ FieldTab<T> fields() const { return copy_fields<T>(6, m1, m2, m3); }
};

// (u_i u_j - B_i B_j) and u x B (:117-134; the momentum and pressure terms are
// linear in NL - MHDNL, so the difference is transformed once).
template <typename T>
struct PhysMHD {
  static constexpr int F_IN = 6, F_OUT = 9;
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
    const T u = in[0], v = in[1], w = in[2], b1 = in[3], b2 = in[4], b3 = in[5];
    out[0] = u * u - b1 * b1;
    out[1] = v * v - b2 * b2;
    out[2] = w * w - b3 * b3;
    out[3] = u * v - b1 * b2;
    out[4] = u * w - b1 * b3;
    out[5] = v * w - b2 * b3;
    out[6] = v * b3 - w * b2;
    out[7] = w * b1 - u * b3;
    out[8] = u * b2 - v * b1;
  }
};

// sums of the MHD products: k_j N_ij (3) and the curl k x X of X = u x B (3)
template <int R, typename T>
__device__ __forceinline__ void acc_mhd(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*D)[R]) {
  T m1[R];
  switch (f) {
    case 6:
      acc_row<R>(k3, v, D[4]);
      acc_row<R>(-k2, v, D[5]);
      break;
    case 7:
      acc_row<R>(-k3, v, D[3]);
      acc_row<R>(k1, v, D[5]);
      break;
    case 8:
#pragma unroll
      for (int r = 0; r < R; ++r) m1[r] = -k1[r];
      acc_row<R>(k2, v, D[3]);
      acc_row<R>(m1, v, D[4]);
      break;
    default:
      acc_sym<R>(f, k1, k2, k3, v, D);
      break;
  }
}

template <typename T>
struct EpiMHD {
  static constexpr int F_IN = 9, NACC = 6;
  static constexpr int X_WARPS64 = 16, X_WARPS32 = 64;  // x_pass_in_registers
  __host__ double io_bytes(long long npts) const {
    return io.bytes(npts, 6) + (force ? (double)sizeof(Cx<T>) * npts * 3 : 0.0);
  }
  StepIO<T> io;
  KTabs<T> k;
  const double *m1, *m2, *m3;
  const Cx<T>* force;  // 3 fields or null
  T nu, eta;
  __device__ __forceinline__ KTabs<T> ktabs() const { return k; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*A)[R]) const {
    acc_mhd<R>(f, k1, k2, k3, v, A);
  }
  struct In {
    StateIn<T, 6> st;
    Cx<T> force[3];
  };
  __device__ __forceinline__ In ld(int i1, int i2, int i3) const {
    const long long s = io.sidx(i1, i2, i3);
    In in;
    in.st.load(io, s);
#pragma unroll
    for (int f = 0; f < 3; ++f) in.force[f] = force ? force[f * io.fstride + s] : mk<T>(0, 0);
    return in;
  }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* A, const In& in) const {
    const long long s = io.sidx(i1, i2, i3);
    const T D = (T)(m1[i1] * m2[i2] * m3[i3]);
    const T kv[3] = {(T)k.k1[i1], (T)k.k2[i2], (T)k.k3[i3]};
    T ksq, ksqi;
    ksq_pair(kv[0], kv[1], kv[2], ksq, ksqi);
    const Cx<T> ph = (-ksqi) * (kv[0] * A[0] + kv[1] * A[1] + kv[2] * A[2]);
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const Cx<T> st = D * in.st.q[f];
      Cx<T> r;
      if (f < 3) {
        r = mul_mi(A[f]) + mik(kv[f], ph) - (nu * ksq) * st;
        r = r + in.force[f];
      } else {
        r = mul_i(A[f]) - (eta * ksq) * st;
      }
      if (io.read_out) io.read_out[f * io.fstride + s] = st;
      io.finish(s, f, D * r, in.st.o[f]);
    }
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
};

// ---- 2x-padded memory closures: t-model, static/dynamic tau-model -----------
// (PySpectral/src/RHSfunctions.py:240-363, :366-497, :592-878)

// 2x-grid index -> N-grid index under unpad_2x (PySpectral/src/padding.py:28-38)
__device__ __forceinline__ int unpad2x_idx(int i, int N) {
  return i < N / 2 ? i : (i >= 2 * N - N / 2 ? i - N : -1);
}
// membership of the resolved set p of seperateModes (PySpectral/src/padding.py:67-79)
__device__ __forceinline__ bool in_p_axis(int i, int N) { return i < N / 2 || i > 2 * N - N / 2; }

// PL on the full 2x grid, split into the q part (inverse-transformed next) and
// unpad_2x(PL) (the resolved RHS).  Optional: the test-filtered Leonard term of
// the dynamic model is stored on the compact G2 box.
template <typename T>
struct EpiPL {
  static constexpr int F_IN = 6, NACC = 3;
  // npts = 2x-grid points: q part written everywhere, resolved state read / PL_p written on the N grid
  __host__ double io_bytes(long long npts) const {
    const double e = (double)sizeof(Cx<T>);
    return e * 3 * npts * (PLfull ? 2.0 : 1.0) + e * 3 * fstride_n * (PLp ? 2.0 : 1.0);
  }
  const Cx<T>* Q;  // N-grid state (3 fields)
  long long fstride_n;
  int N1, N2, N3, n3h;
  int nf2, nf3h;  // 2x-grid sizes: rows_y = 2*N2, k3 count N3+1
  long long fstride_2x;
  KTabs<T> kf;  // 2x-grid wavenumbers
  T nu;
  int rotate;
  T Om1, Om2, Om3;
  const double* filt;  // N-grid test filter per axis (nullptr = no filter): [N1 | N2 | n3h]
  int kfp;             // test-filter split size for the q part (0 = seperateModes)
  Cx<T>* PLq;          // (3, 2N1, 2N2, N3+1)
  Cx<T>* PLp;          // (3, N1, N2, n3h) unpad_2x(PL), may be null
  Cx<T>* Lbox;         // (3, 2kfb-1, 2kfb-1, kfb) Leonard pieces, or null
  int kfb;             // box half-size (test-filter kf)
  Cx<T>* PLfull;       // (3, 2N1, 2N2, N3+1) PL on the whole 2x grid, or null
  __device__ __forceinline__ KTabs<T> ktabs() const { return kf; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*D)[R]) const {
    acc_sym<R>(f, k1, k2, k3, v, D);
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
  struct In {
    Cx<T> u, v, w;
  };
  __device__ __forceinline__ In ld(int i1, int i2, int i3) const {
    const int n1 = unpad2x_idx(i1, N1), n2 = unpad2x_idx(i2, N2);
    const int n3 = i3 < N3 / 2 ? i3 : -1;
    Cx<T> u = mk<T>(0, 0), v = u, w = u;
    // pad_2x(unpad(pad(uhat))) [optionally test-filtered first]
    if (n1 >= 0 && n2 >= 0 && n3 >= 0 && n1 != N1 / 2 && n2 != N2 / 2) {
      const long long s = ((long long)n1 * N2 + n2) * n3h + n3;
      T g = (T)1;
      if (filt) g = (T)(filt[n1] * filt[N1 + n2] * filt[N1 + N2 + n3]);
      u = g * Q[s];
      v = g * Q[fstride_n + s];
      w = g * Q[2 * fstride_n + s];
    }
    return In{u, v, w};
  }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* D, const In& in) const {
    const int n1 = unpad2x_idx(i1, N1), n2 = unpad2x_idx(i2, N2);
    const int n3 = i3 < N3 / 2 ? i3 : -1;
    const Cx<T> u = in.u, v = in.v, w = in.w;
    const T k1 = (T)kf.k1[i1], k2 = (T)kf.k2[i2], k3 = (T)kf.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    Cx<T> ph = (-ksqi) * (k1 * D[0] + k2 * D[1] + k3 * D[2]);
    if (rotate) {
      const Cx<T> cu = Om3 * v - Om2 * w, cv = Om1 * w - Om3 * u, cw = Om2 * u - Om1 * v;
      ph = ph - ((T)2 * ksqi) * mul_i(k1 * cu + k2 * cv + k3 * cw);
    }
    const Cx<T> au = mul_mi(D[0]), av = mul_mi(D[1]), aw = mul_mi(D[2]);
    const Cx<T> pu = au + mik(k1, ph) - (nu * ksq) * u;
    const Cx<T> pv = av + mik(k2, ph) - (nu * ksq) * v;
    const Cx<T> pw = aw + mik(k3, ph) - (nu * ksq) * w;
    bool inp;
    if (kfp > 0) {  // seperateModes_testFilter (PySpectral/src/padding.py:52-64)
      const int M1 = 2 * N1, M2 = 2 * N2;
      inp = (i1 < kfp || i1 >= M1 - kfp + 1) && (i2 < kfp || i2 >= M2 - kfp + 1) && i3 < kfp;
    } else {
      inp = in_p_axis(i1, N1) && in_p_axis(i2, N2) && i3 < N3 / 2;
    }
    const long long s2 = ((long long)i1 * nf2 + i2) * nf3h + i3;
    const Cx<T> z = mk<T>(0, 0);
    PLq[s2] = inp ? z : pu;
    PLq[fstride_2x + s2] = inp ? z : pv;
    PLq[2 * fstride_2x + s2] = inp ? z : pw;
    if (PLfull) {
      PLfull[s2] = pu;
      PLfull[fstride_2x + s2] = pv;
      PLfull[2 * fstride_2x + s2] = pw;
    }
    if (PLp && n1 >= 0 && n2 >= 0 && n3 >= 0) {
      const long long s = ((long long)n1 * N2 + n2) * n3h + n3;
      PLp[s] = pu;
      PLp[fstride_n + s] = pv;
      PLp[2 * fstride_n + s] = pw;
    }
    if (Lbox) {
      // test_filter_2x(-1j k_j (u_i u_j)^ + 1j k_i phat) (PySpectral/src/RHSfunctions.py:813-819)
      const int M1 = 2 * N1, M2 = 2 * N2;
      const int b1 = i1 < kfb ? i1 : (i1 > M1 - kfb ? i1 - M1 + 2 * kfb - 1 : -1);
      const int b2 = i2 < kfb ? i2 : (i2 > M2 - kfb ? i2 - M2 + 2 * kfb - 1 : -1);
      if (b1 >= 0 && b2 >= 0 && i3 < kfb) {
        const int nb = 2 * kfb - 1;
        const long long sb = ((long long)b1 * nb + b2) * kfb + i3;
        const long long fb = (long long)nb * nb * kfb;
        Lbox[sb] = au + pik(k1, ph);
        Lbox[fb + sb] = av + pik(k2, ph);
        Lbox[2 * fb + sb] = aw + pik(k3, ph);
      }
    }
  }
};

// u_j * (PL_q)_i, nine products (PySpectral/src/RHSfunctions.py:325-335)
template <typename T>
struct PhysPLQL {
  static constexpr int F_IN = 6, F_OUT = 9;
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) out[3 * j + i] = in[j] * in[3 + i];
  }
};

// The six symmetric products u_i q_j + u_j q_i (11, 22, 33, 12, 13, 23; 2 u_i q_i
// on the diagonal), q = PL_q: the nine products enter PLQL and its pressure term
// in these sums only (PySpectral/src/RHSfunctions.py:338-352).
template <typename T>
struct PhysPLQS {
  static constexpr int F_IN = 6, F_OUT = 6;
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
#pragma unroll
    for (int i = 0; i < 3; ++i) out[i] = (T)2 * in[i] * in[3 + i];
    out[3] = in[0] * in[4] + in[1] * in[3];
    out[4] = in[0] * in[5] + in[2] * in[3];
    out[5] = in[1] * in[5] + in[2] * in[4];
  }
};

// PLQL on the N grid and the memory-closure RHS = unpad_2x(PL) + coef*PLQL
// (PySpectral/src/RHSfunctions.py:338-358).  With coef_ptr set the PLQL field
// is stored and the RHS is formed later (dynamic tau-model).
template <typename T>
struct EpiPLQL {
  static constexpr int F_IN = 6, NACC = 3;
  __host__ double io_bytes(long long npts) const {
    if (plql_out) return (double)sizeof(Cx<T>) * npts * 3;
    return io.bytes(npts, 3) + (double)sizeof(Cx<T>) * npts * 3;  // + PL_p read
  }
  StepIO<T> io;
  KTabs<T> k;
  const Cx<T>* PLp;
  T coef;
  int rotate;
  T Om1, Om2, Om3;
  int ny1, ny2, ny3;
  Cx<T>* plql_out;  // if non-null: store PLQL and stop
  __device__ __forceinline__ KTabs<T> ktabs() const { return k; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*D)[R]) const {
    acc_sym<R>(f, k1, k2, k3, v, D);
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
  struct In {
    StateIn<T, 3> st;
    Cx<T> pl[3];
  };
  __device__ __forceinline__ In ld(int i1, int i2, int i3) const {
    In in{};
    if (plql_out) return in;
    const long long s = io.sidx(i1, i2, i3);
    in.st.load(io, s);
#pragma unroll
    for (int f = 0; f < 3; ++f) in.pl[f] = PLp[f * io.fstride + s];
    return in;
  }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* D, const In& in) const {
    const long long s = io.sidx(i1, i2, i3);
    const T k1 = (T)k.k1[i1], k2 = (T)k.k2[i2], k3 = (T)k.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    const Cx<T> pt = ksqi * (k1 * D[0] + k2 * D[1] + k3 * D[2]);
    const Cx<T> Lu = mul_mi(D[0]) + pik(k1, pt), Lv = mul_mi(D[1]) + pik(k2, pt), Lw = mul_mi(D[2]) + pik(k3, pt);
    if (plql_out) {
      plql_out[s] = Lu;
      plql_out[io.fstride + s] = Lv;
      plql_out[2 * io.fstride + s] = Lw;
      return;
    }
    Cx<T> u = in.st.q[0], v = in.st.q[1], w = in.st.q[2];
    if (i1 == ny1 || i2 == ny2 || i3 == ny3) u = v = w = mk<T>(0, 0);
    const Cx<T> w0u = coef * Lu, w0v = coef * Lv, w0w = coef * Lw;
    Cx<T> ru = in.pl[0] + w0u, rv = in.pl[1] + w0v, rw = in.pl[2] + w0w;
    if (rotate) {
      ru = ru + (T)2 * (Om3 * v - Om2 * w);
      rv = rv + (T)2 * (Om1 * w - Om3 * u);
      rw = rw + (T)2 * (Om2 * u - Om1 * v);
    }
    if (io.w0_out) {
      io.w0_out[s] = w0u;
      io.w0_out[io.fstride + s] = w0v;
      io.w0_out[2 * io.fstride + s] = w0w;
    }
    if (io.read_out) {
      io.read_out[s] = u;
      io.read_out[io.fstride + s] = v;
      io.read_out[2 * io.fstride + s] = w;
    }
    io.finish(s, 0, ru, in.st.o[0]);
    io.finish(s, 1, rv, in.st.o[1]);
    io.finish(s, 2, rw, in.st.o[2]);
  }
};

// PLQL on the whole 2x grid (the second-order finite memory model needs its
// q part there): the formula of EpiPLQL with the 2x-grid wavenumbers
// (PySpectral/src/RHSfunctions.py:1131-1147), then
//   PLQLq  = seperateModes(PLQL)[1] on the 2x grid (inverse-transformed next),
//   PLQLn  = unpad_2x(PLQL) and PLQLqn = unpad_2x(PLQLq) on the N grid
// (the k3 = N3/2 plane of the N-grid outputs is not written: unpad_2x leaves it zero).
template <typename T>
struct EpiPLQLFull {
  static constexpr int F_IN = 9;
  __host__ double io_bytes(long long npts) const {
    return (double)sizeof(Cx<T>) * (3.0 * npts + 6.0 * fstride_n);
  }
  KTabs<T> kf;  // 2x-grid wavenumbers
  int N1, N2, N3, n3h;
  int nf2, nf3h;
  long long fstride_2x, fstride_n;
  Cx<T>* PLQLq;
  Cx<T>* PLQLn;
  Cx<T>* PLQLqn;
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const {
    const T k1 = (T)kf.k1[i1], k2 = (T)kf.k2[i2], k3 = (T)kf.k3[i3];
    T ksq, ksqi;
    ksq_pair(k1, k2, k3, ksq, ksqi);
    const Cx<T> upu = P[0], upv = P[1], upw = P[2], vpu = P[3], vpv = P[4], vpw = P[5], wpu = P[6],
                wpv = P[7], wpw = P[8];
    const Cx<T> pt = ((T)2 * ksqi) * ((k1 * k1) * upu + (k2 * k2) * vpv + (k3 * k3) * wpw +
                                      (k1 * k2) * (upv + vpu) + (k1 * k3) * (upw + wpu) + (k2 * k3) * (vpw + wpv));
    const Cx<T> L[3] = {
        mik(k1, upu) + mik(k2, vpu) + mik(k3, wpu) + mik(k1, upu) + mik(k2, upv) + mik(k3, upw) + pik(k1, pt),
        mik(k1, upv) + mik(k2, vpv) + mik(k3, wpv) + mik(k1, vpu) + mik(k2, vpv) + mik(k3, vpw) + pik(k2, pt),
        mik(k1, upw) + mik(k2, vpw) + mik(k3, wpw) + mik(k1, wpu) + mik(k2, wpv) + mik(k3, wpw) + pik(k3, pt)};
    const bool inp = in_p_axis(i1, N1) && in_p_axis(i2, N2) && i3 < N3 / 2;
    const long long s2 = ((long long)i1 * nf2 + i2) * nf3h + i3;
    const Cx<T> z = mk<T>(0, 0);
#pragma unroll
    for (int c = 0; c < 3; ++c) PLQLq[c * fstride_2x + s2] = inp ? z : L[c];
    const int n1 = unpad2x_idx(i1, N1), n2 = unpad2x_idx(i2, N2);
    if (n1 >= 0 && n2 >= 0 && i3 < N3 / 2) {
      const long long s = ((long long)n1 * N2 + n2) * n3h + i3;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        PLQLn[c * fstride_n + s] = L[c];
        PLQLqn[c * fstride_n + s] = inp ? z : L[c];
      }
    }
  }
};

// ---- MHD t-model (no reference counterpart) ----------------------------------
// The t-model construction of PySpectral/src/RHSfunctions.py:240-363 applied to
// the MHD operator of PySpectral/src_MPI/RHSfunctions.py:95-175: resolved set
// p = the 2/3-rule set, L evaluated without aliasing on the 2x grid, QL its q
// part, PLQL the linearisation of L about (u, B) in the direction QL.

// Nonlinear MHD operator from the six sums of the nine product spectra
// (acc_mhd): momentum with the pressure projection and the induction curl, as
// in EpiMHD without dissipation, forcing and mask.
template <typename T>
__device__ __forceinline__ void mhd_nonlinear(T k1, T k2, T k3, const Cx<T>* A, Cx<T>* r) {
  T ksq, ksqi;
  ksq_pair(k1, k2, k3, ksq, ksqi);
  const Cx<T> ph = (-ksqi) * (k1 * A[0] + k2 * A[1] + k3 * A[2]);
  r[0] = mul_mi(A[0]) + mik(k1, ph);
  r[1] = mul_mi(A[1]) + mik(k2, ph);
  r[2] = mul_mi(A[2]) + mik(k3, ph);
  r[3] = mul_i(A[3]);
  r[4] = mul_i(A[4]);
  r[5] = mul_i(A[5]);
}

// 2x-grid epilogue: QL = L(u, B) on the modes outside the 2/3-rule set.
template <typename T>
struct EpiMHDQ {
  static constexpr int F_IN = 9, NACC = 6;
  __host__ double io_bytes(long long npts) const { return (double)sizeof(Cx<T>) * 6 * npts; }
  KTabs<T> kf;                 // 2x-grid wavenumbers
  const double *m1, *m2, *m3;  // N-grid 2/3-rule masks
  int N1, N2, n3h;             // N-grid sizes (k3 count N3/2+1)
  int nf2, nf3h;               // 2x-grid rows along y, k3 count
  long long fstride_2x;
  T scale;  // 2x-grid transform sums -> N-grid convention (1/8)
  Cx<T>* QL;  // (6, 2N1, 2N2, N3+1)
  __device__ __forceinline__ KTabs<T> ktabs() const { return kf; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*A)[R]) const {
    acc_mhd<R>(f, k1, k2, k3, v, A);
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
  struct In {};
  __device__ __forceinline__ In ld(int, int, int) const { return In{}; }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* A, const In&) const {
    const int n1 = unpad2x_idx(i1, N1), n2 = unpad2x_idx(i2, N2);
    const bool resolved = n1 >= 0 && n2 >= 0 && i3 < n3h && m1[n1] * m2[n2] * m3[i3] != 0.0;
    const long long s = ((long long)i1 * nf2 + i2) * nf3h + i3;
    Cx<T> r[6];
    if (resolved) {
#pragma unroll
      for (int f = 0; f < 6; ++f) r[f] = mk<T>(0, 0);
    } else {
      mhd_nonlinear((T)kf.k1[i1], (T)kf.k2[i2], (T)kf.k3[i3], A, r);
    }
#pragma unroll
    for (int f = 0; f < 6; ++f) QL[f * fstride_2x + s] = scale * r[f];
  }
};

// Linearised MHD products about (u, B) in the direction (q, r) = QL:
// u_i q_j + q_i u_j - B_i r_j - r_i B_j and q x B + u x r.
template <typename T>
struct PhysMHDLin {
  static constexpr int F_IN = 12, F_OUT = 9;
  __device__ __forceinline__ void operator()(long long, int, const T* in, T* out) const {
    const T u = in[0], v = in[1], w = in[2], b1 = in[3], b2 = in[4], b3 = in[5];
    const T q1 = in[6], q2 = in[7], q3 = in[8], r1 = in[9], r2 = in[10], r3 = in[11];
    out[0] = (T)2 * (u * q1 - b1 * r1);
    out[1] = (T)2 * (v * q2 - b2 * r2);
    out[2] = (T)2 * (w * q3 - b3 * r3);
    out[3] = u * q2 + q1 * v - b1 * r2 - r1 * b2;
    out[4] = u * q3 + q1 * w - b1 * r3 - r1 * b3;
    out[5] = v * q3 + q2 * w - b2 * r3 - r2 * b3;
    out[6] = (q2 * b3 - q3 * b2) + (v * r3 - w * r2);
    out[7] = (q3 * b1 - q1 * b3) + (w * r1 - u * r3);
    out[8] = (q1 * b2 - q2 * b1) + (u * r2 - v * r1);
  }
};

// N-grid epilogue: RHS = (plain MHD RHS, precomputed) + Ct t D PLQL, then the
// RK stage update.
template <typename T>
struct EpiMHDT {
  static constexpr int F_IN = 9, NACC = 6;
  __host__ double io_bytes(long long npts) const {
    return io.bytes(npts, 6) + (double)sizeof(Cx<T>) * 6 * npts + (w0_out ? (double)sizeof(Cx<T>) * 6 * npts : 0.0);
  }
  StepIO<T> io;
  KTabs<T> k;
  const double *m1, *m2, *m3;
  const Cx<T>* rhs6;  // plain MHD RHS (6 fields)
  T coef;             // Ct t / 8 (2x-grid sums -> N-grid convention)
  Cx<T>* w0_out;      // memory term (6 fields) or null
  __device__ __forceinline__ KTabs<T> ktabs() const { return k; }
  template <int R>
  __device__ __forceinline__ void acc(int f, const T* k1, T k2, T k3, const Cx<T>* v, Cx<T> (*A)[R]) const {
    acc_mhd<R>(f, k1, k2, k3, v, A);
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const { epi_point<T>(*this, i1, i2, i3, P); }
  struct In {
    typename StepIO<T>::Old o[6];
    Cx<T> r[6];
  };
  __device__ __forceinline__ In ld(int i1, int i2, int i3) const {
    const long long s = io.sidx(i1, i2, i3);
    In in;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      in.r[f] = rhs6[f * io.fstride + s];
      in.o[f] = io.fetch(s, f, io.mode == kStage1 ? io.Q[f * io.fstride + s] : mk<T>(0, 0));
    }
    return in;
  }
  __device__ __forceinline__ void fin(int i1, int i2, int i3, const Cx<T>* A, const In& in) const {
    const long long s = io.sidx(i1, i2, i3);
    const T D = (T)(m1[i1] * m2[i2] * m3[i3]);
    Cx<T> r[6];
    mhd_nonlinear((T)k.k1[i1], (T)k.k2[i2], (T)k.k3[i3], A, r);
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const Cx<T> w0 = (coef * D) * r[f];
      if (w0_out) w0_out[f * io.fstride + s] = w0;
      io.finish(s, f, in.r[f] + w0, in.o[f]);
    }
  }
};

// Stores the F product spectra.
template <typename T, int F>
struct EpiStore {
  static constexpr int F_IN = F, NACC = 0;  // no sums: put() stores each field's modes as they come
  static constexpr int X_WARPS64 = 2, X_WARPS32 = 2;  // x_pass_in_registers
  Cx<T>* out;
  long long fstride;
  int n2, n3h;
  __host__ double io_bytes(long long npts) const { return (double)sizeof(Cx<T>) * npts * F; }
  __device__ __forceinline__ void put(int f, int i1, int i2, int i3, Cx<T> v) const {
    out[f * fstride + ((long long)i1 * n2 + i2) * n3h + i3] = v;
  }
  __device__ void operator()(int i1, int i2, int i3, const Cx<T>* P) const {
#pragma unroll
    for (int m = 0; m < F; ++m) put(m, i1, i2, i3, P[m]);
  }
};

}  // namespace psb

// ---- learned subgrid closure (no counterpart in the reference) -------------
#include "psb_mlp.cuh"

namespace psb {

// (u,v,w) -> (u,v,w, du_i/dx_j = i k_j u_i for i,j = 1..3), gradient order
// g[3*i + j]; the spectral expander of the learned closure's x-inverse pass.
template <typename T>
struct PreGrad {
  static constexpr int F_SRC = 3, F_DST = 12;
  __device__ void operator()(int i, int o, int c, const AxisArgs<T>& a, const Cx<T>* s, Cx<T>* d) const {
    const T k[3] = {(T)a.k_row[i], (T)a.k_outer[o], (T)a.k_col[c]};
#pragma unroll
    for (int f = 0; f < 3; ++f) d[f] = s[f];
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
      for (int j = 0; j < 3; ++j) d[3 + 3 * f + j] = pik(k[j], s[f]);
  }
};

// y-inverse pass of the velocity-gradient pipeline: the CTA of component q
// (outer index q*M1 + x) reads u_q and its x derivative (fields q and 3+q of
// the x pass) and writes u_q, du_q/dx and du_q/dy = i k_y u_q (fields q, 3+q
// and 6+q): the y derivative is formed on load (derivatives commute with the
// x transform, so the x pass need not carry it) and every source field is
// read once.  GROUPS outer groups; input and output field strides of 3 fields.
template <typename T>
struct PreYGrad {
  static constexpr int F_SRC = 2, F_DST = 3, GROUPS = 3, IN_FIELDS = 3, OUT_FIELDS = 3;
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t;
    t.nf = 3;
    t.sa[1] = 1;
    t.kind[2] = kIkRow;
    return t;
  }
  __device__ void operator()(int i, int, int, const AxisArgs<T>& a, const Cx<T>* s, Cx<T>* d) const {
    d[0] = s[0];
    d[1] = s[1];
    d[2] = pik((T)a.k_row[i], s[0]);
  }
};

// (u,v,w) -> (u,v,w, du_i/dx) on the x-inverse pass; the y-inverse pass
// (PreYGrad) adds du_i/dy and the z-pass forms du_i/dz = i k3 u_i itself, so
// the x pass carries 6 fields and the y pass 9 instead of 12.  z-pass input
// order is PreGrad's: u,v,w then g[3*i + j]; after the y pass the stored
// fields are (u, v, w, ux, vx, wx, uy, vy, wy).
template <typename T>
struct PreGradXY {
  static constexpr int F_SRC = 3, F_DST = 6, F_B = 9, Z_DERIVED = 3;
  __host__ FieldTab<T> fields() const {
    FieldTab<T> t;
    t.nf = 6;
    for (int g = 0; g < 6; ++g) {
      t.sa[g] = (unsigned char)(g % 3);
      t.kind[g] = g < 3 ? kCopy : kIkRow;
    }
    return t;
  }
  using YPass = PreYGrad<T>;
  __device__ void operator()(int i, int, int, const AxisArgs<T>& a, const Cx<T>* s, Cx<T>* d) const {
    const T k1 = (T)a.k_row[i];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
      d[f] = s[f];
      d[3 + f] = pik(k1, s[f]);
    }
  }
  // z-pass input f (0..11) -> stored field and whether it is differentiated along z
  __host__ static void zsrc(int f, int& src, bool& der) {
    if (f < 3) {
      src = f;
      der = false;
      return;
    }
    const int i = (f - 3) / 3, j = (f - 3) % 3;
    der = j == 2;
    src = der ? i : 3 + 3 * j + i;
  }
};

// Products u_i u_j plus the MLP subgrid stress, summed so that one forward
// transform per component carries both: out_ij = u_i u_j + tau_ij / s^2 in the
// reference's real-space scaling (real-space arrays equal physical / s).
// The MLP runs warp-cooperatively on tensor cores over all points of the CTA.
// ACT: the network's hidden activation (kActRelu or kActGelu); a separate
// kernel per activation keeps the ReLU kernel free of the GELU's registers.
// H: the network's hidden width (32 or 64).
template <typename T, int ACT = kActRelu, int H = 64>
struct PhysLearned {
  static constexpr int F_IN = 12, F_OUT = 6;
  static constexpr bool BLOCK = true;
  static constexpr int EXTRA_SMEM = (int)((sizeof(MlpFwdSmem<H>) + 15) / 16 * 16);
  // 4 pencils per CTA by default (3 CTAs per SM at 3N/2 = 96, FP32); the
  // autotuner also tries 8 (fuller transform passes, 2 CTAs per SM)
  static constexpr int DEFAULT_PPC = 4, MAX_PPC = 8;
  const float* params;
  const float* norm;
  T sphys;      // s: physical = real-space * s
  float delta;  // filter width fed to the MLP
  __device__ void setup(unsigned char* extra) const {
    mlp_stage_fwd<H>(*reinterpret_cast<MlpFwdSmem<H>*>(extra), params, norm);
  }
  __device__ void block(const Cx<T>* R, Cx<T>* W, int P, int M, int LS, T fac, long long, long long,
                        unsigned char* extra) const {
    block_act(R, W, P, M, LS, fac, extra);
  }
  // Each warp takes tiles of 16 consecutive points (pencil-major); a lane
  // holds rows g and g+8 of a tile and locates them once per tile.
  __device__ __forceinline__ void block_act(const Cx<T>* R, Cx<T>* W, int P, int M, int LS, T fac,
                                            unsigned char* extra) const {
    const MlpFwdSmem<H>& s = *reinterpret_cast<const MlpFwdSmem<H>*>(extra);
    if ((M & 7) == 0 && (P & 1) == 0) {
      block_tiles(reinterpret_cast<const T*>(R), reinterpret_cast<T*>(W), P, M, LS, fac, s);
      return;
    }
    const int npts = P * M;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nw = blockDim.x >> 5;
    const T is2 = (T)1 / (sphys * sphys);
    const T fs = fac * sphys;
    for (int pt0 = warp * 16; pt0 < npts; pt0 += nw * 16) {
      // rows g and g+8 of the tile: pencil p, position z
      int rp[2], rz[2];
      bool ok[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int pt = pt0 + g + 8 * h;
        ok[h] = pt < npts;
        rp[h] = ok[h] ? pt / M : 0;
        rz[h] = ok[h] ? pt - rp[h] * M : 0;
      }
      auto val = [&](int f, int h) -> T {
        const int r = f * P + rp[h];
        const Cx<T> v = R[(size_t)(r >> 1) * LS + rz[h]];
        return (r & 1) ? v.y : v.x;
      };
      uint32_t xa[4];
      mlp_xfrag(s, xa, [&](int r, int f) -> float {
        const int h = r >= 8 ? 1 : 0;
        if (!ok[h]) return s.xmean[f];
        return f < 9 ? (float)(val(3 + f, h) * fs) : delta;
      });
      float y[4];
      mlp_forward_fast<ACT, H>(s, xa, y);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 2 * t + (e & 1);
        const int h = e < 2 ? 0 : 1;
        if (c >= kMlpOut || !ok[h]) continue;
        const int ii = c < 3 ? c : (c == 5 ? 1 : 0);
        const int jj = c < 3 ? c : (c == 3 ? 1 : 2);
        const T tau = (T)(y[e] * s.ystd[c] + s.ymean[c]);
        const T o = (fac * val(ii, h)) * (fac * val(jj, h)) + tau * is2;
        const int r = c * P + rp[h];
        reinterpret_cast<T*>(W + (size_t)(r >> 1) * LS + rz[h])[r & 1] = o;
      }
    }
  }
  // The same computation when packed lines pair pencils of one field (P even)
  // and M % 8 == 0: real line (f, p) is half p&1 of packed line f*P/2 + p/2
  // (lines LS apart), so field f of pencil p at z is T element
  // f*P*LS + 2((p/2) LS + z) + (p&1).  A tile is 16 consecutive T elements of
  // a packed line -- 8 consecutive z of a pencil pair, both halves -- so the
  // 8 rows a lane group reads are consecutive words and, with the field
  // stride P*LS = 28 (mod 32) words at P = 4 (LS = 7 mod 16), the 32 lanes of a
  // feature gather (8 rows x 4 features) hit 32 different banks.  Each lane keeps the
  // offsets, normalisation and output coefficients of its fragment slots in
  // registers; per tile it computes one base index per row.
  __device__ __forceinline__ void block_tiles(const T* __restrict__ R, T* __restrict__ W, int P, int M, int LS,
                                              T fac, const MlpFwdSmem<H>& s) const {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nw = blockDim.x >> 5;
    const int fst = P * LS;
    const T is2 = (T)1 / (sphys * sphys);
    const T fs = fac * sphys;
    // feature slot q = 2 hk + e holds feature f = 2t + 8hk + e: a gradient
    // (f < 9, physical field 3 + f), the filter width (f = 9) or padding
    int foff[4];
    float fm[4], fi[4], fc[4];
    bool fg[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int f = 2 * t + 8 * (q >> 1) + (q & 1);
      fg[q] = f < 9;
      foff[q] = fg[q] ? (3 + f) * fst : 0;
      fm[q] = f < kMlpIn ? s.xmean[f] : 0.f;
      fi[q] = f < kMlpIn ? s.xistd[f] : 0.f;
      fc[q] = f == 9 ? (delta - s.xmean[f]) * s.xistd[f] : 0.f;
    }
    // output slot e2 = e & 1: column c = 2t + e2 (valid for c < 6) = u_ii u_jj + tau_c / s^2
    int ooff[2], ioff[2], joff[2];
    float ys[2], ym[2];
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      const int c = 2 * t + e2;
      const int ii = c < 3 ? c : (c == 5 ? 1 : 0);
      const int jj = c < 3 ? c : (c == 3 ? 1 : 2);
      ooff[e2] = c * fst;
      ioff[e2] = ii * fst;
      joff[e2] = jj * fst;
      ys[e2] = c < kMlpOut ? s.ystd[c] : 0.f;
      ym[e2] = c < kMlpOut ? s.ymean[c] : 0.f;
    }
    const bool out_ok = t < 3;
    const int tpp = M >> 3, ntile = (P >> 1) * tpp;
    for (int tile = warp; tile < ntile; tile += nw) {
      const int pp = tile / tpp;  // pencil pair
      const int z0 = (tile - pp * tpp) << 3;
      const int b0 = 2 * (pp * LS + z0) + g;  // row g; row g + 8 is b0 + 8
      float v[8];
#pragma unroll
      for (int hr = 0; hr < 2; ++hr)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float x = (float)(R[b0 + 8 * hr + foff[q]] * fs);
          v[hr * 4 + q] = fg[q] ? (x - fm[q]) * fi[q] : fc[q];
        }
      uint32_t xa[4];
      xa[0] = pack_bf16(v[0], v[1]);  // row g,   k 2t..2t+1
      xa[1] = pack_bf16(v[4], v[5]);  // row g+8, k 2t..2t+1
      xa[2] = pack_bf16(v[2], v[3]);  // row g,   k 2t+8..
      xa[3] = pack_bf16(v[6], v[7]);  // row g+8, k 2t+8..
      float y[4];
      mlp_forward_fast<ACT, H>(s, xa, y);
      if (out_ok) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int e2 = e & 1;
          const int b = b0 + 8 * (e >> 1);
          const T tau = (T)(y[e] * ys[e2] + ym[e2]);
          W[b + ooff[e2]] = (fac * R[b + ioff[e2]]) * (fac * R[b + joff[e2]]) + tau * is2;
        }
      }
    }
  }
  // The same computation on the register z pass's buffer (psb_zreg.cuh): slot f
  // holds field f, pencil p's element (i, r) at f*ss + p*LS + i*BP + r, two
  // consecutive real points per element.  Points are taken in storage order, 16
  // per tile; the six results of a point go to slots 6..11 (its own last six
  // gradients, read before the first MMA of the tile).  The inputs are physical
  // already.
  template <int A, int B, int BP, int LS>
  __device__ __forceinline__ void points(T* __restrict__ X, int P, int ss, unsigned char* extra) const {
    const MlpFwdSmem<H>& s = *reinterpret_cast<const MlpFwdSmem<H>*>(extra);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nw = blockDim.x >> 5;
    const int fst = 2 * ss;
    const T is2 = (T)1 / (sphys * sphys);
    int foff[4];
    float fm[4], fi[4], fc[4];
    bool fg[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int f = 2 * t + 8 * (q >> 1) + (q & 1);
      fg[q] = f < 9;
      foff[q] = fg[q] ? (3 + f) * fst : 0;
      fm[q] = f < kMlpIn ? s.xmean[f] : 0.f;
      fi[q] = f < kMlpIn ? s.xistd[f] : 0.f;
      fc[q] = f == 9 ? (delta - s.xmean[f]) * s.xistd[f] : 0.f;
    }
    int ooff[2], ioff[2], joff[2];
    float ys[2], ym[2];
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      const int c = 2 * t + e2;
      const int ii = c < 3 ? c : (c == 5 ? 1 : 0);
      const int jj = c < 3 ? c : (c == 3 ? 1 : 2);
      ooff[e2] = (6 + c) * fst;
      ioff[e2] = ii * fst;
      joff[e2] = jj * fst;
      ys[e2] = c < kMlpOut ? s.ystd[c] : 0.f;
      ym[e2] = c < kMlpOut ? s.ymean[c] : 0.f;
    }
    const int npts = P * A * 2 * B;
    // a warp runs eight or so tiles here: the width-32 network's weights stay in registers
    MlpFrags<H == 32 ? 32 : 16> w;
    if constexpr (H == 32) w.load(s);
    for (int pt0 = warp * 16; pt0 < npts; pt0 += nw * 16) {
      int b[2];
      bool ok[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int pt = pt0 + g + 8 * h;
        ok[h] = pt < npts;
        const int blk = pt / (2 * B), off = pt - blk * (2 * B);
        const int p = blk / A, i = blk - p * A;
        b[h] = ok[h] ? 2 * (p * LS + i * BP) + off : 0;
      }
      float v[8];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float x = (float)(X[b[h] + foff[q]] * sphys);
          v[h * 4 + q] = fg[q] ? (x - fm[q]) * fi[q] : fc[q];
        }
      uint32_t xa[4];
      xa[0] = pack_bf16(v[0], v[1]);
      xa[1] = pack_bf16(v[4], v[5]);
      xa[2] = pack_bf16(v[2], v[3]);
      xa[3] = pack_bf16(v[6], v[7]);
      float y[4];
      if constexpr (H == 32)
        mlp_forward_held<ACT, H>(s, w, xa, y);
      else
        mlp_forward_fast<ACT, H>(s, xa, y);
      if (t < 3) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int e2 = e & 1, h = e >> 1;
          if (!ok[h]) continue;
          const T tau = (T)(y[e] * ys[e2] + ym[e2]);
          X[b[h] + ooff[e2]] = X[b[h] + ioff[e2]] * X[b[h] + joff[e2]] + tau * is2;
        }
      }
    }
  }
};

}  // namespace psb
