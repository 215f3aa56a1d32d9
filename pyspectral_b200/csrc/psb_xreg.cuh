// Register x pass: the last forward transform of the product spectra, fused
// with the spectral epilogue, for the lengths L = A B R of PSB_REG_X.
//
// A CTA owns C columns (64 bytes of k3) of one k2 and takes the F_IN fields one
// after another: radix A from global memory, one shared-memory exchange (two
// with a middle radix B > 1), radix R in the thread that owns the output rows
// j + A B r of a column.  There each field is added to the epilogue's sums
// (acc: NACC accumulators of R modes) and dropped; after the last field the
// thread has everything its modes need and finishes them (fin: projection,
// viscous term, RK stage).
//
// What bounds it: HBM / L2 traffic and the latency of the field loop.  The
// fused pass it replaces staged every field of a column in shared memory (12
// fields: 100 KB, one or two CTAs per SM, six shared-memory accesses per
// element); this one holds two buffers of one field, and the sums instead of
// the products, so more CTAs run per SM.  R is small because NACC R accumulators
// live through the whole loop: with R = 8 an FP64 thread of the t-model needs 228
// registers, two CTAs per SM.  Measured per launch on a B200, before -> after:
//   t-model 128^3 FP64   PLQL 373 -> 127 us, PL (256 points) 547 -> 490
//   DNS 256^3 FP32 (384 points)  1063 -> 482     Smagorinsky 128^3 FP64  267 -> 152
// Launches that leave the SMs few warps pay for the series of fields and run the
// staged pass (x_pass_in_registers): DNS 32^3 FP64 10.5 us.
#pragma once
#include "psb_physics.cuh"

namespace psb {

#define PSB_REG_X(X) \
  X(16, 4, 1, 4)     \
  X(18, 6, 1, 3)     \
  X(24, 6, 1, 4)     \
  X(32, 8, 1, 4)     \
  X(36, 9, 1, 4)     \
  X(48, 12, 1, 4)    \
  X(54, 9, 2, 3)     \
  X(64, 8, 2, 4)     \
  X(72, 6, 3, 4)     \
  X(96, 8, 3, 4)     \
  X(108, 9, 3, 4)    \
  X(128, 8, 4, 4)    \
  X(144, 9, 4, 4)    \
  X(162, 9, 6, 3)    \
  X(192, 8, 6, 4)    \
  X(216, 9, 6, 4)    \
  X(256, 8, 8, 4)    \
  X(288, 9, 8, 4)    \
  X(324, 9, 9, 4)    \
  X(384, 12, 8, 4)   \
  X(432, 12, 9, 4)   \
  X(512, 16, 8, 4)

// Columns per CTA: 64 bytes of a row.
template <typename T>
constexpr int xreg_cols() {
  return 64 / (int)sizeof(Cx<T>);
}
// Threads: one per output item (A B of them per column), whole warps.
template <typename T, int A, int B>
constexpr int xreg_threads() {
  return (A * B * xreg_cols<T>() + 31) / 32 * 32;
}

// S: groups of threads that share a tile's fields (group g takes fields g, g + S,
// ...); the partial sums are exchanged at the end and each group finishes 1/S of
// the rows.  S = 3 is a third of the serial chain (x_groups).
template <typename T, class Epi, int A, int B, int R, int S>
__device__ __forceinline__ void xreg_body(const XEpiArgs<T>& a, const Epi& epi, int bx, int gx) {
  constexpr int L = A * B * R, AB = A * B, C = xreg_cols<T>(), NT = xreg_threads<T, A, B>(), F = Epi::F_IN;
  constexpr int NACC = Epi::NACC;
  pdl_trigger();
  // the blocks of the columns without products come first: they are the longest chain
  const int nextra = gx - a.main_blocks;
  if (bx < nextra) {
    pdl_wait();
    xfwd_epi_extra<T, Epi>(a, epi, a.main_blocks + bx, gx);
    return;
  }
  bx -= nextra;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int grp = S == 1 ? 0 : threadIdx.x / NT, tid = threadIdx.x - grp * NT;
  Cx<T>* X0 = reinterpret_cast<Cx<T>*>(smem_raw);
  Cx<T>* X = X0 + grp * 2 * L * C;
  Cx<T>* Y = X + L * C;
  constexpr int BUFS = S * 2 * L * C, SUMS = S > 1 ? S * NACC * R * AB * C : 0;
  Cx<T>* tb = X0 + (BUFS > SUMS ? BUFS : SUMS);  // W_{AB}^{rk} at r A + k (B > 1)
  const int ntile = (a.kz + C - 1) / C;
  const int o = bx / ntile, c0 = (bx - o * ntile) * C;
  const int c = tid % C, q = tid / C;
  const int col = c0 + c;
  const bool ok = col < a.kz;
  const Cx<T> zero = mk<T>(0, 0);
  const Cx<T>* tw = a.tw + a.plan.tw_off;
  const Cx<T>* src = a.in + (long long)o * a.in_ostride + (ok ? col : 0);
  // the output item's own twiddles, for every field; the middle radix's go to
  // shared memory, k fastest
  Cx<T> wq[R];
#pragma unroll
  for (int r = 1; r < R; ++r) wq[r] = tw[r * (q < AB ? q : 0)];
  if constexpr (B > 1)
    for (int t = threadIdx.x; t < AB; t += S * NT) tb[t] = tw[(t / A) * (t % A) * R];
  // output rows and their k1
  int row[R];
  T k1[R], k2 = 0, k3 = 0;
  Cx<T> D[NACC > 0 ? NACC : 1][R];
#pragma unroll
  for (int r = 0; r < R; ++r) row[r] = q < AB ? row_of(a.out_map, q + AB * r, a.n1) : -1;
  if constexpr (NACC > 0) {
    const KTabs<T> kt = epi.ktabs();
    k2 = (T)kt.k2[o];
    k3 = ok ? (T)kt.k3[col] : (T)0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      k1[r] = row[r] >= 0 ? (T)kt.k1[row[r]] : (T)0;
#pragma unroll
      for (int m = 0; m < NACC; ++m) D[m][r] = zero;
    }
  }
  // radix A: item j = q < L / A = B R (at most A B) reads rows j + (L / A) r; the
  // next field's are in flight while this one goes through the other radices
  static_assert(R <= A, "one load item per thread");
  const bool lead = q < B * R;
  Cx<T> v[A];
  pdl_wait();
  if (lead) {
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = src[grp * a.in_fstride + (long long)(q + L / A * r) * a.in_rstride];
  }
#pragma unroll 1
  for (int it = 0; it < (F + S - 1) / S; ++it) {
    const int f = it * S + grp;
    const bool has = F % S == 0 || f < F;
    Cx<T>* W = B == 1 && (it & 1) ? Y : X;
    if (lead && has) {
      small_dft<T, A, false>(v);
#pragma unroll
      for (int r = 0; r < A; ++r) W[(q * A + r) * C + c] = v[r];
      if (f + S < F) {
        const Cx<T>* p = src + (f + S) * a.in_fstride;
#pragma unroll
        for (int r = 0; r < A; ++r) v[r] = p[(long long)(q + L / A * r) * a.in_rstride];
      }
    }
    __syncthreads();
    if constexpr (B > 1) {
      // radix B: item j < L / B, sub-transforms of length A
      for (int j = q; has && j < L / B; j += NT / C) {
        const int k = j % A;
        Cx<T> u[B];
#pragma unroll
        for (int r = 0; r < B; ++r) u[r] = X[(j + L / B * r) * C + c];
#pragma unroll
        for (int r = 1; r < B; ++r) u[r] = cmul(u[r], tb[r * A + k]);
        small_dft<T, B, false>(u);
#pragma unroll
        for (int r = 0; r < B; ++r) Y[((j - k) * B + k + A * r) * C + c] = u[r];
      }
      __syncthreads();
    }
    if (q < AB && has) {
      const Cx<T>* Z = B == 1 ? W : Y;
      Cx<T> u[R];
#pragma unroll
      for (int r = 0; r < R; ++r) u[r] = Z[(q + AB * r) * C + c];
#pragma unroll
      for (int r = 1; r < R; ++r) u[r] = cmul(u[r], wq[r]);
      small_dft<T, R, false>(u);
      if constexpr (NACC > 0) {
        epi.template acc<R>(f, k1, k2, k3, u, D);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (ok && row[r] >= 0) epi.put(f, row[r], o, col, u[r]);
      }
    }
  }
  if constexpr (NACC > 0) {
    if constexpr (S > 1) {
      // sums of rows r = g (mod S) to group g
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < NACC; ++m)
          if (q < AB && r % S != grp) X0[((grp * NACC + m) * R + r) * (AB * C) + q * C + c] = D[m][r];
      __syncthreads();
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int g = 0; g < S; ++g)
#pragma unroll
          for (int m = 0; m < NACC; ++m)
            if (q < AB && r % S == grp && g != grp)
              D[m][r] = D[m][r] + X0[((g * NACC + m) * R + r) * (AB * C) + q * C + c];
    }
    // a mode's loads (FP32: two modes') ahead of its stores
    constexpr int G = sizeof(T) == 4 && S == 1 ? 2 : 1;
    if (ok) {
#pragma unroll
      for (int r0 = 0; r0 < R; r0 += G) {
        typename Epi::In in[G];
#pragma unroll
        for (int u = 0; u < G; ++u)
          if (r0 + u < R && row[(r0 + u) % R] >= 0 && (S == 1 || r0 % S == grp))
            in[u] = epi.ld(row[(r0 + u) % R], o, col);
#pragma unroll
        for (int u = 0; u < G; ++u) {
          if (r0 + u >= R || row[(r0 + u) % R] < 0 || !(S == 1 || r0 % S == grp)) continue;
          Cx<T> Ds[NACC];
#pragma unroll
          for (int m = 0; m < NACC; ++m) Ds[m] = D[m][(r0 + u) % R];
          epi.fin(row[(r0 + u) % R], o, col, Ds, in[u]);
        }
      }
    }
  }
  if (!ok || grp != 0) return;
  // output rows without a position carry no products
  const int zlo = a.out_map.lo, zhi = min(a.out_map.hi, a.n1);
  for (int i = zlo + q; i < zhi; i += NT / C) {
    Cx<T> P[F];
#pragma unroll
    for (int f = 0; f < F; ++f) P[f] = zero;
    epi(i, o, col, P);
  }
}

// CTAs per SM the registers are bounded for: 128 registers a thread (168 from four
// FP64 sums on), in FP32 104 (128 from four sums on).  One CTA more where it is the
// second and leaves 72 registers (FP64 with four sums: 128), or in FP32 the third of
// seven or more warps and leaves 96; up to four sums.  The blocks are large, one CTA is
// a third to a half of an SM.  Measured, one CTA per SM -> two
// (or two -> three at 108 points): FP32 DNS 192 points 80 -> 60 us (128^3), 216
// points 111 -> 86 (144^3), 108 points 23 -> 17 (72^3); Smagorinsky 144 points
// 76 -> 47 (96^3), 192 points 138 -> 107 (128^3).  With six sums the epilogues
// spill instead, as do blocks of six warps in threes (18 warps are five on a
// scheduler, 96 registers): two there in launches of no more blocks (MANY false; DNS
// 64^3 FP32 38.4 -> 36.2 us a right-hand side), three in larger ones (64 x 288 x 64
// 147 -> 136) and in batches.
template <typename T, class Epi, int A, int B, int R, bool MANY>
constexpr int xreg_minb() {
  constexpr int nt = xreg_threads<T, A, B>();
  constexpr int regs = sizeof(T) == 8 ? (Epi::NACC > 3 ? 168 : 128) : (Epi::NACC > 3 ? 128 : 104);
  constexpr int b = 65536 / (regs * nt), left = 65536 / ((b + 1) * nt);
  constexpr bool more = sizeof(T) == 8 ? Epi::NACC == 4 && b == 1 && left >= 128
                                       : Epi::NACC <= 4 && ((b == 1 && left >= 72) || (b == 2 && nt >= 224 && left >= 96));
  if (!MANY && sizeof(T) == 4 && nt == 192 && b == 3) return 2;
  return more ? (b < 16 ? b + 1 : 16) : (b < 1 ? 1 : (b > 16 ? 16 : b));
}

// Shared memory: two buffers a group, or the sums that the groups exchange where
// those are larger (NACC / 2 times the buffers), and the middle radix's twiddles.
template <typename T, class Epi, int A, int B, int R, int S>
constexpr size_t xreg_smem() {
  const int bufs = S * 2 * A * B * R * xreg_cols<T>(), sums = S > 1 ? S * Epi::NACC * R * A * B * xreg_cols<T>() : 0;
  return (size_t)((bufs > sums ? bufs : sums) + (B > 1 ? A * B : 0)) * sizeof(Cx<T>);
}

// grid = main_blocks + extra (main block b: column tile b % ntile, outer b / ntile)
template <typename T, class Epi, int A, int B, int R, int S, bool MANY>
__global__ void __launch_bounds__(S* xreg_threads<T, A, B>(), xreg_minb<T, Epi, A, B, R, MANY>() / S > 0
                                                                   ? xreg_minb<T, Epi, A, B, R, MANY>() / S
                                                                   : 1)
    xreg_kernel(const __grid_constant__ XEpiArgs<T> a, const __grid_constant__ Epi epi) {
  xreg_body<T, Epi, A, B, R, S>(a, epi, blockIdx.x, gridDim.x);
}

// Batched: grid = (main_blocks + extra, runs); run blockIdx.y reads A[y], epi[y].
template <typename T, class Epi, int A, int B, int R>
__global__ void __launch_bounds__(xreg_threads<T, A, B>(), xreg_minb<T, Epi, A, B, R, true>())
    xreg_batch(const XEpiArgs<T>* __restrict__ args, const Epi* __restrict__ epi, int main_blocks) {
  XEpiArgs<T> a = args[blockIdx.y];
  a.main_blocks = main_blocks;
  xreg_body<T, Epi, A, B, R, 1>(a, epi[blockIdx.y], blockIdx.x, gridDim.x);
}

}  // namespace psb
