// Register z pass: c2r of the F_IN spectral pencils, the physical-space
// products, r2c of the F_OUT results, for the real lengths M = 2 A B of
// PSB_REG_Z_F32 / _F64, with the transforms and the products in registers.
//
// A real pencil of M points is one complex transform of H = M/2 = A B points
// of z[n] = x[2n] + i x[2n+1]; with X[k], k <= H, its spectrum and W = e^{2 pi i/M},
//   inverse: Z[k] = (X[k] + conj X[H-k]) + i W^k (X[k] - conj X[H-k])
//   forward: X[k] = (Z[k] + conj Z[H-k])/2 - (i/2) W^{-k} (Z[k] - conj Z[H-k]).
// The complex transform runs as two radices around one shared-memory exchange:
//   outer item (line, j)   the A elements k = j + B s of a line, one lane per j;
//                          the other half of each pair, H - k = (B-j) + B (A-1-s),
//                          is register A-1-s of lane B-j of the same group of B
//                          lanes and comes over with a warp shuffle (lane 0 pairs
//                          with its own register A-s).  Radix A, element (i, j).
//   middle item (pencil, i) the B points n = i + A r of EVERY field of a pencil:
//                          radix B of the inverse, the products of those points,
//                          radix B of the forward transform, written back into
//                          the thread's own elements.
//   outer item again       radix A, the pairing, the store of the kept k3.
// Inverse and forward twiddles W_H^{ij} are the middle thread's own (i is
// fixed), so they are registers shared by every field.  Shared memory sees one
// write and one read per element and direction, against five and five plus the
// twiddles in the staged form (psb_passes.cuh), and one buffer instead of two.
//
// What bounds it: shared-memory bandwidth and the issue rate in the small
// grids, HBM beyond L2.  The line stride and the stride of i are chosen at
// compile time for the fewest bank conflicts of the two access patterns.
// Measured per launch on a B200, staged form -> this one:
//   Smagorinsky FP64   64^3 77 -> 50 us, 128^3 650 -> 400
//   t-model 128^3 FP64 (256 points)   products 1304 -> 371, PLQL 1767 -> 511
//   MHD t-model 128^3 FP32            815 -> 312 and 1294 -> 493
//   DNS 256^3 FP32 (384 points)       2320 -> 462
//   Smagorinsky FP32, 162 points      121 -> 50
//   learned FP32       64^3 50 -> 48, 128^3 352 -> 292 (the network's MMAs remain)
//
// Fields sit in `slots` of the buffer (slot, pencil, i, j); Mid<Phys> says
// which slot an input or output field uses: an output may reuse the slot of an
// input once the thread has read it for the last time.
#pragma once
#include "psb_physics.cuh"

namespace psb {

template <class F, int... I>
__device__ __forceinline__ void sfor_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant 0), ..., f(integral_constant N-1)
template <int N, class F>
__device__ __forceinline__ void sfor(F&& f) {
  sfor_impl(f, std::make_integer_sequence<int, N>{});
}

// Strides of the exchange buffer, in complex elements: element (i, j) of a
// line at i*bp + j, lines ls apart.  The pair with the fewest bank conflicts
// over the outer access (lanes: j fastest, then lines, whole lines per warp) and the middle access
// (lanes: i fastest, then pencils); banks = complex elements per 128 bytes.
struct ZStrides {
  int bp, ls;
};
constexpr int z_conflicts(int A, int B, int bp, int ls, int banks) {
  int cost = 0;
  for (int w = 0; w < 2; ++w) {  // middle, outer
    for (int g = 0; g < 64 / banks; ++g) {
      int n[16] = {}, worst = 0;
      for (int l = 0; l < banks; ++l) {
        const int t = g * banks + l, lane = t % 32;
        int a = 0;
        if (w == 0) {
          a = (t / A) * ls + (t % A) * bp;
        } else {
          if (lane >= 32 / B * B) continue;
          a = (t / 32 * (32 / B) + lane / B) * ls + lane % B;
        }
        const int b = a % banks;
        if (++n[b] > worst) worst = n[b];
      }
      cost += worst;
    }
  }
  return cost;
}
constexpr ZStrides z_strides(int A, int B, int banks) {
  ZStrides best{B, A * B};
  int bc = 1 << 30;
  for (int bp = B; bp <= B + 2; ++bp)
    for (int pad = 0; pad < banks; ++pad) {
      const int ls = A * bp + pad;
      const int c = z_conflicts(A, B, bp, ls, banks) * 64 + (bp - B) * A + pad;
      if (c < bc) {
        bc = c;
        best = ZStrides{bp, ls};
      }
    }
  return best;
}

template <typename T, int A_, int B_>
struct ZPlan {
  static constexpr int A = A_, B = B_, H = A * B, M = 2 * H;
  static constexpr ZStrides S = z_strides(A, B, 128 / (int)sizeof(Cx<T>));
  static constexpr int BP = S.bp, LS = S.ls;
  static constexpr int NT = 128, GW = 32 / B;  // threads; lines per warp of the outer stages
  // CTAs per SM: 128 registers (FP64) or 96 (FP32) per thread; the large radices need more
  static constexpr int REGS = A * (int)sizeof(Cx<T>) / 4;  // of an outer item's elements
  // (heavy: of a physics that holds more than four fields of a point)
  static constexpr int minb(int heavy) {
    const int b = sizeof(T) == 8 ? (REGS > 64 ? 3 : 4) : (REGS > 48 ? 4 : 5);
    return heavy == 0 || B <= 4 ? b : (heavy == 1 ? (sizeof(T) == 8 ? 3 : 4) : (sizeof(T) == 8 ? 2 : 3));
  }
};

// What a middle item sees: its points of the field in a slot.
template <typename T, int A, int B>
struct MidIO {
  Cx<T>* base;  // element (i, 0) of slot 0
  int ss;       // slot stride
  Cx<T> w[B];  // W_H^{ij} = exp(-2 pi i ij / H)
  // inverse radix B of a slot: unnormalised physical values at n = i + A r
  __device__ __forceinline__ void load(int slot, Cx<T>* v) const {
    const Cx<T>* p = base + slot * ss;
#pragma unroll
    for (int j = 0; j < B; ++j) v[j] = p[j];
#pragma unroll
    for (int j = 1; j < B; ++j) v[j] = cmul(v[j], conjg(w[j]));
    small_dft<T, B, true>(v);
  }
  // forward radix B of physical values, left in a slot
  __device__ __forceinline__ void store(int slot, Cx<T>* v) const {
    Cx<T>* p = base + slot * ss;
    small_dft<T, B, false>(v);
    p[0] = v[0];
#pragma unroll
    for (int j = 1; j < B; ++j) p[j] = cmul(v[j], w[j]);
  }
};

// pointwise products of two physical fields (both points of every element)
template <typename T>
__device__ __forceinline__ Cx<T> had(Cx<T> a, Cx<T> b) { return mk<T>(a.x * b.x, a.y * b.y); }
template <typename T>
__device__ __forceinline__ Cx<T> had_add(Cx<T> a, Cx<T> b, Cx<T> c) { return mk<T>(a.x * b.x + c.x, a.y * b.y + c.y); }
template <typename T>
__device__ __forceinline__ Cx<T> had_sub(Cx<T> a, Cx<T> b, Cx<T> c) { return mk<T>(c.x - a.x * b.x, c.y - a.y * b.y); }

// Mid<Phys>: the middle stage of a physics functor.  The physical fields are 1/fac
// times the physics' arguments: every result is quadratic in them (|S| S_ij
// included), so fac^2 is applied with the forward transform's own factor when the
// results are stored.  fac is between 0.7 and 1.5, the power of two next to the whole
// normalisation being in the stored fields already (field_scale).
//   SLOTS        slots of the buffer
//   HEAVY        how many more than four fields' points a thread holds (0, 1, 2)
//   DERIV        1: some inputs are z derivatives (ZArgs::dz), 2: or means (ZArgs::in2)
//   JOBS         independent sets of fields, each a tile of its own: job k takes
//                fields [in0(k), in0(k+1)) to results [out0(k), out0(k+1))
//   in(f), out(g) slot of an input / output field
//   run<A, B>(phys, io, job)
template <class Phys>
struct Mid {
  static constexpr bool value = false;
};
// one job of every field
template <class Phys>
struct MidOneJob {
  static constexpr int JOBS = 1, DERIV = 0;
  __host__ __device__ static constexpr int in0(int k) { return k == 0 ? 0 : Phys::F_IN; }
  __host__ __device__ static constexpr int out0(int k) { return k == 0 ? 0 : Phys::F_OUT; }
};

// six products of (u, v, w): two fields in registers at a time
template <typename T>
struct MidProducts {
  // slots: u 0, v 1, w 2; uu -> 3, vv -> 5, ww -> 2, uv -> 4, uw -> 0, vw -> 1
  __host__ __device__ static constexpr int out(int g) { return g == 0 ? 3 : (g == 1 ? 5 : (g == 2 ? 2 : (g == 3 ? 4 : (g == 4 ? 0 : 1)))); }
  template <int A, int B>
  __device__ static __forceinline__ void run(const MidIO<T, A, B>& io) {
    Cx<T> u[B], v[B], p[B];
    io.load(0, u);
    io.load(1, v);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had(u[r], u[r]);
    io.store(3, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had(u[r], v[r]);
    io.store(4, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had(v[r], v[r]);
    io.store(5, p);
    if constexpr (B * sizeof(Cx<T>) <= 128) {  // u stays in registers
      Cx<T> w[B];
      io.load(2, w);
#pragma unroll
      for (int r = 0; r < B; ++r) v[r] = had(v[r], w[r]);
      io.store(1, v);
#pragma unroll
      for (int r = 0; r < B; ++r) u[r] = had(u[r], w[r]);
      io.store(0, u);
#pragma unroll
      for (int r = 0; r < B; ++r) w[r] = had(w[r], w[r]);
      io.store(2, w);
    } else {  // u is read again
      io.load(2, u);
#pragma unroll
      for (int r = 0; r < B; ++r) v[r] = had(v[r], u[r]);
      io.store(1, v);
#pragma unroll
      for (int r = 0; r < B; ++r) p[r] = had(u[r], u[r]);
      io.store(2, p);
      io.load(0, v);
#pragma unroll
      for (int r = 0; r < B; ++r) v[r] = had(u[r], v[r]);
      io.store(0, v);
    }
  }
};

template <typename T>
struct Mid<PhysProducts<T>> : MidOneJob<PhysProducts<T>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 6, HEAVY = 0;
  __host__ __device__ static constexpr int in(int f) { return f; }
  __host__ __device__ static constexpr int out(int g) { return MidProducts<T>::out(g); }
  template <int A, int B>
  __device__ static __forceinline__ void run(const PhysProducts<T>&, const MidIO<T, A, B>& io, int) {
    MidProducts<T>::template run<A, B>(io);
  }
};

// products (job 0) and the Smagorinsky stress (job 1)
template <typename T>
struct Mid<PhysSmag<T>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 6, JOBS = 2, HEAVY = 0, DERIV = 2;
  __host__ __device__ static constexpr int in0(int k) { return k == 0 ? 0 : (k == 1 ? 3 : 9); }
  __host__ __device__ static constexpr int out0(int k) { return 6 * k; }
  __host__ __device__ static constexpr int in(int f) { return f < 3 ? f : f - 3; }
  __host__ __device__ static constexpr int out(int g) { return g < 6 ? MidProducts<T>::out(g) : g - 6; }
  template <int A, int B>
  __device__ static __forceinline__ void run(const PhysSmag<T>& phys, const MidIO<T, A, B>& io, int job) {
    if (job == 0) {
      MidProducts<T>::template run<A, B>(io);
      return;
    }
    Cx<T> q[B];  // S:S, then -2 nu_t
#pragma unroll
    for (int r = 0; r < B; ++r) q[r] = mk<T>(0, 0);
    if constexpr (B * sizeof(Cx<T>) <= 32) {
      Cx<T> s[6][B];
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        io.load(m, s[m]);
        const T c = m < 3 ? (T)1 : (T)2;
#pragma unroll
        for (int r = 0; r < B; ++r) q[r] = had_add(c * s[m][r], s[m][r], q[r]);
      }
      nut(phys, q, std::integral_constant<int, B>{});
#pragma unroll
      for (int m = 0; m < 6; ++m) {
#pragma unroll
        for (int r = 0; r < B; ++r) s[m][r] = had(q[r], s[m][r]);
        io.store(m, s[m]);
      }
    } else {  // the six strains do not fit the registers: read twice
      Cx<T> s[B];
#pragma unroll 1
      for (int m = 0; m < 6; ++m) {
        io.load(m, s);
        const T c = m < 3 ? (T)1 : (T)2;
#pragma unroll
        for (int r = 0; r < B; ++r) q[r] = had_add(c * s[r], s[r], q[r]);
      }
      nut(phys, q, std::integral_constant<int, B>{});
#pragma unroll 1
      for (int m = 0; m < 6; ++m) {
        io.load(m, s);
#pragma unroll
        for (int r = 0; r < B; ++r) s[r] = had(q[r], s[r]);
        io.store(m, s);
      }
    }
  }
  template <int B>
  __device__ static __forceinline__ void nut(const PhysSmag<T>& phys, Cx<T>* q, std::integral_constant<int, B>) {
    const T c = (T)-2 * phys.csd2 * (T)1.4142135623730950488;
#pragma unroll
    for (int r = 0; r < B; ++r) q[r] = mk<T>(c * sqrt(q[r].x), c * sqrt(q[r].y));
  }
};

// u_i u_j - B_i B_j and u x B: two of the three components of (u, B) in
// registers at a time; component 0 is read again for its products with 2
template <typename T>
struct Mid<PhysMHD<T>> : MidOneJob<PhysMHD<T>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 9, HEAVY = 1;
  __host__ __device__ static constexpr int in(int f) { return f; }
  // out 0..8 -> slots 6, 7, 2, 8, 0, 4, 5, 3, 1
  __host__ __device__ static constexpr int out(int g) {
    return g == 0 ? 6 : (g == 1 ? 7 : (g == 2 ? 2 : (g == 3 ? 8 : (g == 4 ? 0 : (g == 5 ? 4 : (g == 6 ? 5 : (g == 7 ? 3 : 1)))))));
  }
  template <int A, int B>
  __device__ static __forceinline__ void run(const PhysMHD<T>&, const MidIO<T, A, B>& io, int) {
    Cx<T> u[B], b[B], v[B], d[B], p[B];
    io.load(0, u);
    io.load(3, b);
    io.load(1, v);
    io.load(4, d);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(b[r], b[r], had(u[r], u[r]));
    io.store(6, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(d[r], d[r], had(v[r], v[r]));
    io.store(7, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(b[r], d[r], had(u[r], v[r]));
    io.store(8, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(v[r], b[r], had(u[r], d[r]));  // u b2 - v b1
    io.store(1, p);
    io.load(2, u);  // w, b3
    io.load(5, b);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(b[r], b[r], had(u[r], u[r]));
    io.store(2, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(d[r], b[r], had(v[r], u[r]));
    io.store(4, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(u[r], d[r], had(v[r], b[r]));  // v b3 - w b2
    io.store(5, p);
    io.load(0, v);  // u, b1
    io.load(3, d);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(d[r], b[r], had(v[r], u[r]));  // u w - b1 b3
    io.store(0, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_sub(v[r], b[r], had(u[r], d[r]));  // w b1 - u b3
    io.store(3, p);
  }
};

// nine products u_j q_i: u in registers, one q at a time
template <typename T>
struct Mid<PhysPLQL<T>> : MidOneJob<PhysPLQL<T>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 9, HEAVY = 1;
  __host__ __device__ static constexpr int in(int f) { return f; }
  // out 3 j + i = u_j q_i: q_0 -> slots 0, 1, 2; q_1 -> 3, 6, 7; q_2 -> 4, 5, 8
  __host__ __device__ static constexpr int slot(int j, int i) {
    return i == 0 ? j : (i == 1 ? (j == 0 ? 3 : 5 + j) : (j == 0 ? 4 : (j == 1 ? 5 : 8)));
  }
  __host__ __device__ static constexpr int out(int g) { return slot(g / 3, g % 3); }
  template <int A, int B>
  __device__ static __forceinline__ void run(const PhysPLQL<T>&, const MidIO<T, A, B>& io, int) {
    Cx<T> u[3][B], q[B], p[B];
#pragma unroll
    for (int j = 0; j < 3; ++j) io.load(j, u[j]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      io.load(3 + i, q);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
#pragma unroll
        for (int r = 0; r < B; ++r) p[r] = had(u[j][r], q[r]);
        io.store(slot(j, i), p);
      }
    }
  }
};

// symmetric products of u and q: two of the three components of (u, q) in
// registers at a time; component 0 is read again for its product with 2
template <typename T>
struct Mid<PhysPLQS<T>> : MidOneJob<PhysPLQS<T>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 7, HEAVY = 1;
  __host__ __device__ static constexpr int in(int f) { return f; }
  // out 11, 22, 33, 12, 13, 23 -> slots 1, 6, 2, 4, 0, 5
  __host__ __device__ static constexpr int out(int g) {
    return g == 0 ? 1 : (g == 1 ? 6 : (g == 2 ? 2 : (g == 3 ? 4 : (g == 4 ? 0 : 5))));
  }
  template <int A, int B>
  __device__ static __forceinline__ void run(const PhysPLQS<T>&, const MidIO<T, A, B>& io, int) {
    Cx<T> u[B], q[B], v[B], w[B], p[B];
    io.load(0, u);
    io.load(3, q);
    io.load(1, v);
    io.load(4, w);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = (T)2 * had(u[r], q[r]);
    io.store(1, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_add(u[r], w[r], had(v[r], q[r]));
    io.store(4, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = (T)2 * had(v[r], w[r]);
    io.store(6, p);
    io.load(2, u);
    io.load(5, q);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_add(u[r], w[r], had(v[r], q[r]));
    io.store(5, p);
    io.load(0, v);
    io.load(3, w);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = (T)2 * had(u[r], q[r]);
    io.store(2, p);
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = had_add(u[r], w[r], had(v[r], q[r]));
    io.store(0, p);
  }
};

// linearised MHD products: two components of (u, B, q, r) in registers at a
// time; component 0 is read again for its products with 2
template <typename T>
struct Mid<PhysMHDLin<T>> : MidOneJob<PhysMHDLin<T>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 12, HEAVY = 2;
  __host__ __device__ static constexpr int in(int f) { return f; }
  // out 0..8 -> slots 1, 4, 2, 7, 0, 5, 8, 3, 10
  __host__ __device__ static constexpr int out(int g) {
    return g == 0 ? 1 : (g == 1 ? 4 : (g == 2 ? 2 : (g == 3 ? 7 : (g == 4 ? 0 : (g == 5 ? 5 : (g == 6 ? 8 : (g == 7 ? 3 : 10)))))));
  }
  // component c of (u, B, q, r)
  template <int A, int B>
  __device__ static __forceinline__ void comp(const MidIO<T, A, B>& io, int c, Cx<T> (*x)[B]) {
#pragma unroll
    for (int m = 0; m < 4; ++m) io.load(3 * m + c, x[m]);
  }
  // 2 (u q - b r) of one component
  template <int A, int B>
  __device__ static __forceinline__ void diag(const MidIO<T, A, B>& io, int slot, Cx<T> (*x)[B]) {
    Cx<T> p[B];
#pragma unroll
    for (int r = 0; r < B; ++r) p[r] = (T)2 * had_sub(x[1][r], x[3][r], had(x[0][r], x[2][r]));
    io.store(slot, p);
  }
  // u_a q_b + q_a u_b - b_a r_b - r_a b_b
  template <int A, int B>
  __device__ static __forceinline__ void sym(const MidIO<T, A, B>& io, int slot, Cx<T> (*x)[B], Cx<T> (*y)[B]) {
    Cx<T> p[B];
#pragma unroll
    for (int r = 0; r < B; ++r)
      p[r] = had_sub(x[3][r], y[1][r], had_sub(x[1][r], y[3][r], had_add(x[2][r], y[0][r], had(x[0][r], y[2][r]))));
    io.store(slot, p);
  }
  // (q_a b_b - q_b b_a) + (u_a r_b - u_b r_a)
  template <int A, int B>
  __device__ static __forceinline__ void cross(const MidIO<T, A, B>& io, int slot, Cx<T> (*x)[B], Cx<T> (*y)[B]) {
    Cx<T> p[B];
#pragma unroll
    for (int r = 0; r < B; ++r)
      p[r] = had_sub(y[2][r], x[1][r], had(x[2][r], y[1][r])) + had_sub(y[0][r], x[3][r], had(x[0][r], y[3][r]));
    io.store(slot, p);
  }
  template <int A, int B>
  __device__ static __forceinline__ void run(const PhysMHDLin<T>&, const MidIO<T, A, B>& io, int) {
    Cx<T> x[4][B], y[4][B];
    comp(io, 0, x);
    comp(io, 1, y);
    diag(io, 1, x);
    diag(io, 4, y);
    sym(io, 7, x, y);
    cross(io, 10, x, y);
    comp(io, 2, x);
    diag(io, 2, x);
    sym(io, 5, y, x);
    cross(io, 8, y, x);
    comp(io, 0, y);
    sym(io, 0, y, x);
    cross(io, 3, x, y);
  }
};

// The learned closure: the network runs over the tile's points between an
// inverse and a forward middle stage (PhysLearned::points); tau and the
// products of a point replace its last six gradients (slots 6..11).
template <typename T, int ACT, int HID>
struct Mid<PhysLearned<T, ACT, HID>> : MidOneJob<PhysLearned<T, ACT, HID>> {
  static constexpr bool value = true;
  static constexpr int SLOTS = 12, HEAVY = 0, DERIV = 1;
  __host__ __device__ static constexpr int in(int f) { return f; }
  __host__ __device__ static constexpr int out(int g) { return 6 + g; }
};

// Element k of the inverse's complex spectrum from a = X[k] and y = X[H-k]
// (HA, HY: known to be non-zero), w = exp(-2 pi i k / M).
template <bool HA, bool HY, typename T>
__device__ __forceinline__ Cx<T> z_inv_one(Cx<T> a, Cx<T> y, Cx<T> w) {
  if constexpr (HA && HY) {
    const Cx<T> d = cmul(mk<T>(a.x - y.x, a.y + y.y), conjg(w));
    return mk<T>(a.x + y.x - d.y, a.y - y.y + d.x);
  } else if constexpr (HA) {
    const Cx<T> d = cmul(a, conjg(w));
    return mk<T>(a.x - d.y, a.y + d.x);
  } else {
    const Cx<T> d = cmul(conjg(y), conjg(w));  // minus (X[k] - conj X[H-k]) W^k
    return mk<T>(y.x + d.y, -y.y - d.x);
  }
}
// X[k] of the forward transform, times 2 h: a = Z[k], y = Z[H-k]
template <typename T>
__device__ __forceinline__ Cx<T> z_fwd_one(Cx<T> a, Cx<T> y, Cx<T> w, T h) {
  const Cx<T> d = cmul(mk<T>(a.x - y.x, a.y + y.y), w);
  return mk<T>(h * (a.x + y.x + d.y), h * (a.y - y.y - d.x));
}
template <typename T>
__device__ __forceinline__ Cx<T> shfl(Cx<T> v, int src) {
  return mk<T>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
// x[s] <- one(x[s], its pair) over the first NOUT of the A elements of an outer
// item, of which the first NIN are non-zero: the pair of s is register A-1-s of
// lane `partner`, or for column 0 the lane's own register A-s (y0 for s = 0).
// Called by whole warps.
template <typename T, int A, int NIN, int NOUT, class One>
__device__ __forceinline__ void z_pair_all(Cx<T>* x, Cx<T> y0, bool col0, int partner, One one) {
  Cx<T> prev = y0;
  sfor<(A + 1) / 2>([&](auto ic) {
    constexpr int s = decltype(ic)::value, t = A - 1 - s;
    // the pair of s: register t of a lane, or A - s (zero with t when NIN <= t; s = 0: y0)
    constexpr bool ls = s < NIN, lt = t < NIN, ps = lt || (s == 0 && NIN == A), pt = ls || s + 1 < NIN;
    const Cx<T> lo = x[s], hi = x[t];
    Cx<T> ylo = mk<T>(0, 0), yhi = ylo;
    if constexpr (s < NOUT && ps) {
      const Cx<T> plo = shfl(hi, partner);
      ylo = col0 ? prev : plo;
    }
    if constexpr (s != t && t < NOUT && pt) {
      const Cx<T> phi = shfl(lo, partner);
      yhi = col0 ? x[s + 1] : phi;
    }
    if constexpr (s != t && t < NOUT)
      x[t] = one(hi, yhi, std::integral_constant<int, t>{}, std::integral_constant<bool, lt>{},
                 std::integral_constant<bool, pt>{});
    if constexpr (s < NOUT)
      x[s] = one(lo, ylo, ic, std::integral_constant<bool, ls>{}, std::integral_constant<bool, ps>{});
    prev = hi;
  });
}

// Slot stride: lines of P pencils.  A block physics gathers 8 consecutive reals
// of 4 pairs of fields per instruction: 2 (mod 4) elements spread them over the
// 32 banks.
template <class Phys, typename T, int A, int B>
__host__ __device__ inline int z_slot_stride(int P) {
  int ss = P * ZPlan<T, A, B>::LS;
  if (phys_is_block<Phys>::value)
    while ((ss & 7) != 2 && (ss & 7) != 6) ++ss;
  return ss;
}
template <class Phys, typename T, int A, int B>
__host__ inline size_t z_reg_smem(int P) {
  return ((size_t)A * B + (size_t)Mid<Phys>::SLOTS * z_slot_stride<Phys, T, A, B>(P)) * sizeof(Cx<T>) +
         (phys_is_block<Phys>::value ? phys_is_block<Phys>::extra + 16 : 0);
}
template <class Phys, typename T, int A, int B>
__device__ __forceinline__ unsigned char* z_reg_extra(unsigned char* smem, int P) {
  const size_t o = ((size_t)A * B + (size_t)Mid<Phys>::SLOTS * z_slot_stride<Phys, T, A, B>(P)) * sizeof(Cx<T>);
  return smem + ((o + 15) & ~(size_t)15);
}

// Per-thread constants of a CTA.
template <typename T, int A, int B>
struct ZThread {
  int j, l0, partner;  // outer: column, line of the first round, lane of column B - j
  bool lane_ok;        // the lane belongs to a line (the last 32 mod B lanes do not)
  int i, q0;           // middle: index, first pencil (or (field, pencil))
  const Cx<T>* e;      // exp(-2 pi i (j + B s) / M) at e[B s], in shared memory
};

// P32: 3/2-padded lines: k3 < M/3 stored on either side, A a multiple of three,
// so that the outer elements s < 2A/3 are exactly the stored ones
template <typename T, class Phys, int A, int B, bool P32>
__device__ __forceinline__ void z_reg_tile(const ZArgs<T>& a, const Phys& phys, const ZThread<T, A, B>& th,
                                           MidIO<T, A, B>& io, Cx<T>* buf, unsigned char* extra, int P, int ss,
                                           long long tile, int job) {
  using Pl = ZPlan<T, A, B>;
  using Md = Mid<Phys>;
  constexpr int H = Pl::H, BP = Pl::BP, LS = Pl::LS, NT = Pl::NT;
  const int f0 = Md::in0(job), g0 = Md::out0(job), FI = Md::in0(job + 1) - f0, FO = Md::out0(job + 1) - g0;
  constexpr int LW = NT / 32 * Pl::GW;  // lines per round of the outer stages
  const Cx<T> zero = mk<T>(0, 0);
  const long long p0 = tile * P;
  const int j = th.j;
  const bool col0 = j == 0;
  constexpr int NZ = P32 ? 2 * A / 3 : A;  // stored elements of an outer item
  // ---- outer, inverse (every lane of a warp runs every round: the shuffles need
  // them; lanes without a line repeat the last one and store nothing)
  for (int lb = 0; lb < FI * P; lb += LW) {
    const int l = min(lb + th.l0, FI * P - 1);
    const bool act = th.lane_ok && lb + th.l0 < FI * P;
    const int fl = l / P, p = l - fl * P, f = f0 + fl;
    const long long pen = min(p0 + p, a.npencils - 1);
    const Cx<T>* src = a.in[f] + pen * a.in_pstride[f] + j;
    const int kz = a.in_kz[f] - j;
    Cx<T> x[A], xh = zero;
#pragma unroll
    for (int s = 0; s < A; ++s) x[s] = (P32 ? s < NZ : B * s < kz) ? src[B * s] : zero;
    if (!P32 && col0 && kz > H) xh = src[H];
    if constexpr (Md::DERIV > 0) {
      if (a.dz[f]) {
        // the derivative along z of the stored field
#pragma unroll
        for (int s = 0; s < NZ; ++s) {
          const T k = P32 || B * s < kz ? (T)a.k3[j + B * s] : (T)0;
          x[s] = mk<T>(-k * x[s].y, k * x[s].x);
        }
        if (!P32 && col0 && kz > H) xh.x = -(T)a.k3[H] * xh.y;
      }
    }
    if constexpr (Md::DERIV > 1) {
      if (a.in2[f]) {
        const Cx<T>* s2 = a.in2[f] + pen * a.in_pstride[f] + j;
#pragma unroll
        for (int s = 0; s < NZ; ++s)
          if (P32 || B * s < kz) x[s] = (T)0.5 * (x[s] + s2[B * s]);
        if (!P32 && col0 && kz > H) xh.x = (T)0.5 * (xh.x + s2[H].x);
      }
    }
    // k = 0 and H enter with their real parts (c2r convention)
    if (col0) x[0].y = (T)0;
    xh.y = (T)0;
    z_pair_all<T, A, NZ, A>(x, xh, col0, th.partner, [&](Cx<T> v, Cx<T> y, auto sc, auto ha, auto hy) {
      return z_inv_one<decltype(ha)::value, decltype(hy)::value>(v, y, th.e[B * decltype(sc)::value]);
    });
    small_dft<T, A, true>(x);
    if (act) {
      Cx<T>* Z = buf + Md::in(f) * ss + p * LS + j;
#pragma unroll
      for (int i = 0; i < A; ++i) Z[i * BP] = x[i];
    }
  }
  __syncthreads();
  // ---- middle
  if constexpr (phys_is_block<Phys>::value) {
    Cx<T> v[B];
    if (th.q0 < NT / A)
      for (int q = th.q0; q < FI * P; q += NT / A) {
        const int f = q / P, p = q - f * P;
        io.base = buf + p * LS + th.i * BP;
        io.load(Md::in(f), v);
#pragma unroll
        for (int r = 0; r < B; ++r) io.base[Md::in(f) * ss + r] = a.fac * v[r];
      }
    __syncthreads();
    phys.template points<A, B, BP, LS>(reinterpret_cast<T*>(buf), P, ss, extra);
    __syncthreads();
    if (th.q0 < NT / A)
      for (int q = th.q0; q < FO * P; q += NT / A) {
        const int g = q / P, p = q - g * P;
        io.base = buf + p * LS + th.i * BP;
#pragma unroll
        for (int r = 0; r < B; ++r) v[r] = io.base[Md::out(g) * ss + r];
        io.store(Md::out(g), v);
      }
  } else {
    if (th.q0 < NT / A)
      for (int p = th.q0; p < P; p += NT / A) {
        io.base = buf + p * LS + th.i * BP;
        Md::template run<A, B>(phys, io, job);
      }
  }
  __syncthreads();
  // ---- outer, forward
  const T h = phys_is_block<Phys>::value ? (T)0.5 : (T)0.5 * a.fac * a.fac;
  for (int lb = 0; lb < FO * P; lb += LW) {
    const int l = min(lb + th.l0, FO * P - 1);
    const bool act = th.lane_ok && lb + th.l0 < FO * P;
    const int gl = l / P, p = l - gl * P, g = g0 + gl;
    const Cx<T>* Z = buf + Md::out(g) * ss + p * LS + j;
    Cx<T> x[A];
#pragma unroll
    for (int i = 0; i < A; ++i) x[i] = Z[i * BP];
    small_dft<T, A, false>(x);
    const T xh = (T)2 * h * (x[0].x - x[0].y);  // X[H] in column 0
    z_pair_all<T, A, A, NZ>(x, x[0], col0, th.partner, [&](Cx<T> v, Cx<T> y, auto sc, auto, auto) {
      return z_fwd_one(v, y, th.e[B * decltype(sc)::value], h);
    });
    if (act && p0 + p < a.npencils) {
      const int kzo = a.out_kz - j;
      Cx<T>* dst = a.out[g] + (p0 + p) * a.out_pstride[g] + j;
#pragma unroll
      for (int s = 0; s < NZ; ++s)
        if (P32 || B * s < kzo) dst[B * s] = x[s];
      if (!P32 && col0 && kzo > H) dst[H] = mk<T>(xh, (T)0);
    }
  }
}

// per-thread constants; tw: the table exp(-2 pi i k / M)
template <typename T, int A, int B>
__device__ __forceinline__ void z_reg_thread(const Cx<T>* __restrict__ tw, Cx<T>* etab, int ss, ZThread<T, A, B>& th,
                                             MidIO<T, A, B>& io) {
  using Pl = ZPlan<T, A, B>;
  const int lane = threadIdx.x & 31, grp = lane / B;
  th.j = lane - grp * B;
  th.l0 = (threadIdx.x >> 5) * Pl::GW + grp;
  th.lane_ok = grp < Pl::GW;
  th.partner = th.j == 0 ? lane : grp * B + B - th.j;
  th.i = threadIdx.x % A;
  th.q0 = threadIdx.x / A;
  for (int k = threadIdx.x; k < A * B; k += Pl::NT) etab[k] = tw[k];
  th.e = etab + th.j;
  io.ss = ss;
  io.w[0] = mk<T>(1, 0);
#pragma unroll
  for (int j = 1; j < B; ++j) io.w[j] = tw[2 * th.i * j];
}

// Persistent: tiles of P pencils blockIdx.x, + gridDim.x, ...
template <typename T, class Phys, int A, int B, bool P32>
__global__ void __launch_bounds__(ZPlan<T, A, B>::NT, ZPlan<T, A, B>::minb(Mid<Phys>::HEAVY)) zreg_kernel(const __grid_constant__ ZArgs<T> a, Phys phys,
                                                                     int P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<T>* etab = reinterpret_cast<Cx<T>*>(smem_raw);
  Cx<T>* buf = etab + A * B;
  const int ss = z_slot_stride<Phys, T, A, B>(P);
  unsigned char* extra = z_reg_extra<Phys, T, A, B>(smem_raw, P);
  ZThread<T, A, B> th;
  MidIO<T, A, B> io;
  pdl_trigger();
  z_reg_thread<T, A, B>(a.tw + a.plan.tw_off, etab, ss, th, io);
  if constexpr (phys_is_block<Phys>::value) phys.setup(extra);
  __syncthreads();
  pdl_wait();
  constexpr int NJ = Mid<Phys>::JOBS;
  const long long nitems = (a.npencils + P - 1) / P * NJ;
  for (long long t = blockIdx.x; t < nitems; t += gridDim.x) {
    z_reg_tile<T, Phys, A, B, P32>(a, phys, th, io, buf, extra, P, ss, t / NJ, (int)(t % NJ));
    __syncthreads();
  }
}

// Batched (3/2-padded), persistent over (run, tile); every run has the same shape.
template <typename T, class Phys, int A, int B>
__global__ void __launch_bounds__(ZPlan<T, A, B>::NT, ZPlan<T, A, B>::minb(Mid<Phys>::HEAVY))
    zreg_batch(const ZArgs<T>* __restrict__ args, const Phys* __restrict__ phys, int runs, int P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<T>* etab = reinterpret_cast<Cx<T>*>(smem_raw);
  Cx<T>* buf = etab + A * B;
  const int ss = z_slot_stride<Phys, T, A, B>(P);
  unsigned char* extra = z_reg_extra<Phys, T, A, B>(smem_raw, P);
  ZThread<T, A, B> th;
  MidIO<T, A, B> io;
  pdl_trigger();
  z_reg_thread<T, A, B>(args[0].tw + args[0].plan.tw_off, etab, ss, th, io);
  __syncthreads();
  constexpr int NJ = Mid<Phys>::JOBS;
  const long long ntiles = (args[0].npencils + P - 1) / P * NJ;  // per run
  int staged = -1;
  for (long long it = blockIdx.x; it < ntiles * runs; it += gridDim.x) {
    const int r = (int)(it / ntiles);
    if (r != staged) {
      if constexpr (phys_is_block<Phys>::value) phys[r].setup(extra);
      if (staged < 0) pdl_wait();
      staged = r;
    }
    const Phys ph = phys[r];
    z_reg_tile<T, Phys, A, B, true>(args[r], ph, th, io, buf, extra, P, ss, (it - r * ntiles) / NJ,
                                    (int)((it - r * ntiles) % NJ));
    __syncthreads();  // the next item (or the next run's staging) reuses the shared memory
  }
}

// H = M/2 -> A, B.  The middle radix B decides the registers of the products
// (B elements of two to eight fields), the outer radix A of the pairing (2 A
// elements); FP64 takes the smaller of either.
#define PSB_REG_Z_F32(X) \
  X(12, 3, 4)            \
  X(16, 4, 4)            \
  X(18, 6, 3)            \
  X(24, 6, 4)            \
  X(27, 9, 3)            \
  X(32, 8, 4)            \
  X(36, 9, 4)            \
  X(48, 12, 4)           \
  X(54, 9, 6)            \
  X(64, 16, 4)           \
  X(72, 9, 8)            \
  X(81, 9, 9)            \
  X(96, 12, 8)           \
  X(108, 18, 6)          \
  X(128, 16, 8)          \
  X(144, 18, 8)          \
  X(162, 18, 9)          \
  X(192, 24, 8)          \
  X(216, 27, 8)          \
  X(256, 32, 8)
#define PSB_REG_Z_F64(X) \
  X(12, 3, 4)            \
  X(16, 4, 4)            \
  X(18, 6, 3)            \
  X(24, 6, 4)            \
  X(27, 9, 3)            \
  X(32, 8, 4)            \
  X(36, 9, 4)            \
  X(48, 12, 4)           \
  X(54, 9, 6)            \
  X(64, 16, 4)           \
  X(72, 12, 6)           \
  X(81, 9, 9)            \
  X(96, 12, 8)           \
  X(108, 18, 6)          \
  X(128, 16, 8)          \
  X(144, 18, 8)          \
  X(162, 18, 9)          \
  X(192, 24, 8)

}  // namespace psb
