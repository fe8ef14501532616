// Device-side building blocks shared by the h2b200 CUDA sources (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "h2b200_internal.h"

#define H2B_CUDA_TRY(call)                                                                     \
  do {                                                                                        \
    cudaError_t err__ = (call);                                                               \
    if (err__ != cudaSuccess) {                                                               \
      h2b_set_error("%s:%d: %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(err__));  \
      return H2B_ERR_CUDA;                                                                    \
    }                                                                                         \
  } while (0)

// Counts kernel launches made by the library (every host thread), read with h2b_launch_count.
// Each direct launch site of the assembly, classification and matvec kernels calls it once.
void h2b_note_launch(void);

// 1/(4 pi): constant of the fundamental solutions of Laplace and Helmholtz
// (KERNEL_CONST_LAPLACEBEM3D, Library/laplacebem3d.c:33; KERNEL_CONST_HELMHOLTZBEM3D,
// Library/helmholtzbem3d.c:25).
#define H2B_KERNEL_CONST 0.0795774715459476679

// One triangle as the quadrature kernels read it: 128 bytes, 16-byte aligned, loaded with eight
// 16-byte vector loads.  Vertices are in the triangle's own order (H2Lib's gr->t[i]).
struct __align__(16) TriRec {
  double a[3], b[3], c[3];  // vertex coordinates
  double n[3];              // unit normal
  double g;                 // Gram determinant = 2 * area
  uint32_t v[3];            // vertex ids
  uint32_t pad0;
  double pad1;
};
static_assert(sizeof(TriRec) == 128, "TriRec must be 128 bytes");

// A triangle's part of the q = 2 distant rule: its four points, each with its component along the
// unit normal, the normal, the Gram determinant and the vertex ids; 22 words of 8 bytes.
struct __align__(16) QuadRec {
  double p[4][4];  // x, y, z, <p, n>
  double n[3], g;
  uint32_t v[3], pad;
};
static_assert(sizeof(QuadRec) == 176, "QuadRec must be 176 bytes");

// A triangle referenced by a nearfield tile: its id and the local output row/column index of each
// of its three vertices (linear basis) or of the triangle itself in l[0] (constant basis); -1 when
// the vertex is outside the tile.
struct TriRef {
  uint32_t t;
  int16_t l[3];
  int16_t slots;  // local vertex in slot 0, 1, 2 (two bits each), see h2b_triref
};
static_assert(sizeof(TriRef) == 12, "TriRef must be 12 bytes");

// Reciprocal square root in FP64, full precision.
// Seed: the FP64 approximate reciprocal square root instruction (rsqrt.approx.ftz.f64, relative
// error below 1e-6 measured on B200).  One step of Householder's method of third order for
// x^{-1/2}: with e = 1 - x y^2 the root is y (1 - e)^{-1/2} = y (1 + e/2 + 3 e^2/8 + O(e^3)), so a
// seed error of 1e-6 leaves 5/2 (1e-6)^3, far below one rounding: at most 0.51 ulp from 1/sqrt over
// 4M arguments in [1e-12, 64] (two Newton-Raphson steps: 0.99 ulp).  The kernels around it are bound
// by FP64 instructions, five here where two Newton steps take eight: dense constant-basis single
// layer of 8192 triangles 1.23 -> 1.07 ms, linear-basis V and K nearfield of 32768 triangles
// 6.83 -> 6.66 ms (bound by its scatter).  Inputs are squared distances of quadrature points:
// positive and normal.
__device__ __forceinline__ double rsqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y * y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// Lagrange polynomial mu of the nodes xi[0..m) at x, prod_{l != mu} (x - xi_l) / (xi_mu - xi_l)
// (the one-dimensional factor of the tensor interpolation, Library/bem3d.c:8497).
__device__ __forceinline__ double lagrange_1d(double x, const double *xi, int mu, int m) {
  double v = 1.0;
  for (int l = 0; l < m; l++)
    if (l != mu) v *= (x - xi[l]) / (xi[mu] - xi[l]);
  return v;
}

// Allow kernel K up to H2B_MAX_DYN_SMEM bytes of dynamic shared memory, once per process
// (thread-safe static initialisation).  Launches pass the size they need; the attribute never
// changes afterwards, so launches from several host threads (a solve server's workers) cannot
// race on it.
#define H2B_MAX_DYN_SMEM (200u * 1024u)
template <auto K>
inline cudaError_t h2b_allow_smem() {
  static const cudaError_t rc = cudaFuncSetAttribute(
      K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) H2B_MAX_DYN_SMEM);
  return rc;
}

struct dcomplex {
  double re, im;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
