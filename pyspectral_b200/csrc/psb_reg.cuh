// Register passes: the strided-axis passes of the padded transforms for the
// lengths L = A B of PSB_REG_AXIS, with global memory on both sides and one
// shared-memory exchange between the two radices.
//
// Thread (j, c) loads the A elements j + B s of column c straight from the
// input rows (padding and the pointwise factor of the field applied on load),
// runs the radix-A transform, multiplies by the twiddles W_L^{ij} and leaves
// element (i, j) in shared memory; thread (i, c) reads its B elements, runs the
// radix-B transform and stores output positions i + A r.  Consecutive threads
// hold consecutive columns, so every global and shared access of a half-warp
// covers 128 contiguous bytes, and the whole pass costs one write and one read
// of shared memory per element and one barrier.
//
// What bounds it: HBM / L2 traffic.  A CTA is one column tile of one field
// (128 bytes of columns), 100-400 threads with no staging of its own, so several CTAs
// share an SM and their loads cover each other's barrier; the passes it
// replaces kept a tile of every field of a column in one CTA (up to 100 KB of
// shared memory, two CTAs per SM) and made five to seven shared-memory round
// trips per element.  Measured per launch on a B200, before -> after:
//   t-model 128^3 FP64, 256 points  x-inverse 167 -> 42 us, y-inverse 318 -> 68,
//                                   y-forward 439 -> 284
//   DNS 256^3 FP32, 384 points      x-inverse 529 -> 149, y-inverse 894 -> 208
//   learned 128^3 FP32, 192 points  y-inverse 177 -> 87
// FP64 runs at up to 5.7 TB/s of the measured 6.5; FP32 at 2.3 to 4.5, its accesses
// being 8 bytes a thread.
#pragma once
#include "psb_passes.cuh"

namespace psb {

// Lengths with a register pass and their radices.  A >= B: the load side
// (radix A) runs with B threads per column, the store side with A.
#define PSB_REG_AXIS(X) \
  X(16, 4, 4)           \
  X(18, 6, 3)           \
  X(24, 6, 4)           \
  X(32, 8, 4)           \
  X(36, 6, 6)           \
  X(48, 8, 6)           \
  X(54, 9, 6)           \
  X(64, 8, 8)           \
  X(72, 9, 8)           \
  X(96, 12, 8)          \
  X(108, 12, 9)         \
  X(128, 16, 8)         \
  X(144, 12, 12)        \
  X(162, 18, 9)         \
  X(192, 16, 12)        \
  X(216, 18, 12)        \
  X(256, 16, 16)        \
  X(288, 18, 16)        \
  X(324, 18, 18)        \
  X(384, 24, 16)        \
  X(432, 24, 18)        \
  X(512, 32, 16)

// Columns per CTA: 128 bytes of a row.
template <typename T>
constexpr int reg_cols() {
  return 128 / (int)sizeof(Cx<T>);
}

template <typename T, int A, int B, bool INV>
__device__ __forceinline__ void axis_reg_body(const AxisArgs<T>& a, const FieldTab<T>& ft, int bx, int o, int g) {
  constexpr int C = reg_cols<T>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cx<T>* X = reinterpret_cast<Cx<T>*>(smem_raw);
  const int c = threadIdx.x % C, q = threadIdx.x / C;
  const int col = bx * C + c;
  const bool ok = col < a.ncols;
  const Cx<T> zero = mk<T>(0, 0);
  const Cx<T>* tw = a.tw + a.plan.tw_off;
  pdl_trigger();
  pdl_wait();
  if (q < B) {
    const int j = q;
    const Cx<T>* src = a.in + (long long)o * a.in_ostride + ft.sa[g] * a.in_fstride + col;
    Cx<T> v[A];
#pragma unroll
    for (int s = 0; s < A; ++s) {
      const int i = row_of(a.in_map, j + B * s, a.in_rows);
      v[s] = (ok && i >= 0) ? src[(long long)i * a.in_rstride] : zero;
    }
    if (ft.m1 && g >= ft.mfrom) {
      const double mc = ok ? ft.m2[o] : 0.0, m3 = ok ? ft.m3[col] : 0.0;
#pragma unroll
      for (int s = 0; s < A; ++s) {
        const int i = row_of(a.in_map, j + B * s, a.in_rows);
        v[s] = (i >= 0 ? (T)(ft.m1[i] * mc * m3) : (T)0) * v[s];
      }
    }
    if (ft.f1) {
      const double mc = ok ? ft.f2[o] : 0.0, m3 = ok ? ft.f3[col] : 0.0;
#pragma unroll
      for (int s = 0; s < A; ++s) {
        const int i = row_of(a.in_map, j + B * s, a.in_rows);
        v[s] = (i >= 0 ? (T)(ft.f1[i] * mc * m3) : (T)0) * v[s];
      }
    }
    if (ft.kind[g] != kCopy) {
#pragma unroll
      for (int s = 0; s < A; ++s) {
        const int i = row_of(a.in_map, j + B * s, a.in_rows);
        const T k = i >= 0 ? (T)a.k_row[i] : (T)0;
        v[s] = mk<T>(-k * v[s].y, k * v[s].x);
      }
    }
    if (ft.kind[g] == kIkMean) {
      const Cx<T>* src2 = src + (ft.sb[g] - ft.sa[g]) * a.in_fstride;
#pragma unroll
      for (int s = 0; s < A; ++s) {
        const int i = row_of(a.in_map, j + B * s, a.in_rows);
        v[s] = (T)0.5 * (v[s] + ((ok && i >= 0) ? src2[(long long)i * a.in_rstride] : zero));
      }
    }
    small_dft<T, A, INV>(v);
#pragma unroll
    for (int i = 0; i < A; ++i) {
      if (i > 0) {
        Cx<T> w = tw[i * j];
        if (INV) w.y = -w.y;
        v[i] = cmul(v[i], w);
      }
      X[(i * B + j) * C + c] = v[i];
    }
  }
  __syncthreads();
  Cx<T>* dst = a.out + (long long)o * a.out_ostride + g * a.out_fstride + col;
  if (q < A && ok) {
    const int i = q;
    Cx<T> v[B];
#pragma unroll
    for (int j = 0; j < B; ++j) v[j] = X[(i * B + j) * C + c];
    small_dft<T, B, INV>(v);
#pragma unroll
    for (int r = 0; r < B; ++r) {
      const int row = row_of(a.out_map, i + A * r, a.out_rows);
      if (row >= 0) dst[(long long)row * a.out_rstride] = a.scale * v[r];
    }
  }
  // output rows the map leaves without a position are zero
  const int zlo = a.out_map.lo, zhi = min(a.out_map.hi, a.out_rows);
  if (ok)
    for (int row = zlo + q; row < zhi; row += A) dst[(long long)row * a.out_rstride] = zero;
}

// CTAs per SM the registers are bounded for: the A elements of a load item and
// about 36 (FP64: 56) more.
template <typename T, int A>
constexpr int axis_reg_minb() {
  constexpr int regs = A * (int)sizeof(Cx<T>) / 4 + (sizeof(T) == 4 ? 36 : 56);
  constexpr int nt = (A * reg_cols<T>() + 31) / 32 * 32;
  constexpr int b = 65536 / (regs * nt);
  return b < 1 ? 1 : (b > 16 ? 16 : b);
}

// grid = (ceil(ncols / C), nouter, fields); block = A C threads
template <typename T, int A, int B, bool INV>
__global__ void __launch_bounds__(A* reg_cols<T>(), axis_reg_minb<T, A>()) axis_reg_kernel(const __grid_constant__ AxisArgs<T> a,
                                                                    const __grid_constant__ FieldTab<T> ft) {
  axis_reg_body<T, A, B, INV>(a, ft, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Batched: grid.x = column tiles * runs (run-major); run r reads its arguments from args[r].
template <typename T, int A, int B, bool INV>
__global__ void __launch_bounds__(A* reg_cols<T>(), axis_reg_minb<T, A>()) axis_reg_batch(const AxisArgs<T>* __restrict__ args,
                                                                   const __grid_constant__ FieldTab<T> ft) {
  const int nt = (args[0].ncols + reg_cols<T>() - 1) / reg_cols<T>();
  const int run = blockIdx.x / nt;
  axis_reg_body<T, A, B, INV>(args[run], ft, blockIdx.x - run * nt, blockIdx.y, blockIdx.z);
}

}  // namespace psb
