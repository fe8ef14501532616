// H2 matrix-vector product y += alpha A x on the device (sm_100a).
//
// Follows addeval_h2matrix_avector (Library/h2matrix.c:1269):
//   forward transform   xt_t = V_t^T x_t (leaves), xt_t = sum_s E_s^T xt_s (Library/clusterbasis.c:524)
//   coupling / near     yt_t += S_b xt_s,  y_t += N_b x_s      (fastaddeval, Library/h2matrix.c:1211)
//   backward transform  yt_s += E_s yt_t,  y_t += V_t yt_t     (Library/clusterbasis.c:749)
// The nested transforms are multiplied out once after assembly (flatbasis.cu): for every cluster
// t of an admissible block, W_t = V_t (leaf) or [W_s E_s] over the sons s, the |t| x k basis on
// t's own indices, stored transposed (k x |t|).  The forward transform is then xt_t = W_t^T x_t
// and the backward transform y_t += W_t yt_t for every such cluster independently.
//
// Every product is a list of small dense GEMV work items (h2mvm.h: MvItem), ordered by kind and
// run by three launches of one persistent kernel between a gather (xp = x[idx], accumulators
// cleared) and a scatter (y[idx] += alpha yp):
//   1. forward     xt_t += (W_t^T slice) x_slice,   and nearfield   y_r += N_b x_c
//   2. coupling    yt_r += S_b xt_c
//   3. backward    y_slice += (W_t^T slice)^T yt_t
// Vectors are kept in cluster order, so every item's x and y are contiguous slices.  (Running
// all three in one launch, with counters per cluster carrying the dependences, measured slower:
// the counter and claim atomics cost more than the two launch boundaries.)
//
// The kernel streams each item's panel — a contiguous column-major block of N, S or W^T — and its
// x slice into a ring of shared-memory stages with bulk asynchronous copies (cp.async.bulk
// global -> shared, completion counted on an mbarrier per stage), issued by a producer warp, so
// that several panels per SM are in flight while consumer warps multiply earlier ones from
// shared memory.  The copies are local to this GPU and have no cluster multicast.  Every wait is
// bounded: on time-out the kernel sets the plan's error flag, waits (bounded) for its copies in
// flight and returns.  Partial sums reach their outputs with FP64 atomics.
// CX: complex coefficients (Helmholtz) — S, N, x, y complex (interleaved); W real.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "device_common.cuh"
#include "h2mvm.h"

namespace {

constexpr int MAXTHREADS = 288;              // up to 8 consumer warps and the producer warp
constexpr int MAXROWS = 128;                 // rows of an untransposed item (four 32-lane slots)
constexpr uint32_t WAIT_LIMIT = 1u << 24;    // try_wait polls before a stage counts as lost

// Vectors of a product with nrhs right-hand sides.  With a mask (batched solves on a forest:
// mask[surface + r * nseg] for column r) an item skips the columns whose system is done.
struct MvmVecs {
  double *xp, *yp, *xt, *yt;      // work vectors, column r at r * stride
  size_t sxp, syp, sxt, syt;
  uint32_t nrhs, nseg;
  const uint32_t *mask;           // NULL: every column
};

__device__ __forceinline__ bool col_on(const uint32_t *mask, uint32_t nseg, uint32_t seg,
                                       uint32_t r) {
  return !mask || mask[seg + r * nseg] != 0;
}

// xp = x[idx] per column; the accumulators yp, xt, yt are cleared.
template <bool CX>
__global__ void gather_zero_kernel(const double *__restrict__ x, size_t ldx,
                                   const uint32_t *__restrict__ idx, uint32_t n, MvmVecs v,
                                   size_t nyp, size_t nxt, size_t nyt) {
  const size_t i0 = blockIdx.x * (size_t) blockDim.x + threadIdx.x, st = (size_t) gridDim.x * blockDim.x;
  for (uint32_t r = 0; r < v.nrhs; r++) {
    const double *xr = x + r * ldx;
    double *xp = v.xp + r * v.sxp;
    for (size_t i = i0; i < n; i += st) {
      const uint32_t j = idx[i];
      if (CX) {
        xp[2 * i] = xr[2 * j];
        xp[2 * i + 1] = xr[2 * j + 1];
      } else {
        xp[i] = xr[j];
      }
    }
    for (size_t i = i0; i < nyp; i += st) v.yp[r * v.syp + i] = 0.0;
    for (size_t i = i0; i < nxt; i += st) v.xt[r * v.sxt + i] = 0.0;
    for (size_t i = i0; i < nyt; i += st) v.yt[r * v.syt + i] = 0.0;
  }
}

// y[idx[i]] += alpha * yp[i] per column
template <bool CX>
__global__ void scatter_multi_kernel(MvmVecs v, const uint32_t *__restrict__ idx,
                                     double *__restrict__ y, size_t ldy, uint32_t n, double ar,
                                     double ai) {
  for (uint32_t r = 0; r < v.nrhs; r++) {
    const double *yp = v.yp + r * v.syp;
    double *yr = y + r * ldy;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      const uint32_t j = idx[i];
      if (CX) {
        const double re = yp[2 * i], im = yp[2 * i + 1];
        yr[2 * j] += ar * re - ai * im;
        yr[2 * j + 1] += ar * im + ai * re;
      } else {
        yr[j] += ar * yp[i];
      }
    }
  }
}

// One launch of the item kernel.
struct MvLaunch {
  const MvItem *items;
  uint32_t n;
  const void *A[4];        // panel array per kind: W_c^T, N, S, W_r^T (N, S complex when CX)
  const double *X[4];      // x work vector per kind
  double *Y[4];            // y work vector per kind
  size_t sx[4], sy[4];     // column strides (doubles)
  uint32_t first;          // the launch's items: first .. first + n - 1 of the list
  uint32_t nrhs, nseg;
  const uint32_t *mask;
  int *err;
  uint32_t stage_bytes;    // bytes per stage (multiple of 128)
  uint32_t panel_bytes;    // panel region of a stage; the x slices of every column follow
  uint32_t xcol_bytes;     // bytes per x slice of one column (multiple of 16, with slack)
  uint32_t group;          // columns multiplied together (several columns: balanced groups)
  uint32_t run;            // coupling: consecutive panels per warp
  uint32_t x2_doubles;     // coupling: doubles per column of a warp's row slices
  uint32_t stages;         // ring stages, a multiple of nw: stage s belongs to consumer warp s % nw
  uint32_t nw;             // consumer warps; warp nw produces
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t) __cvta_generic_to_shared(p);
}

__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t spin = 0; spin < WAIT_LIMIT; spin++)
    if (bar_try(bar, parity)) return true;
  return false;
}

// [lo, lo + bytes): the 16-byte aligned span that covers [addr, addr + n); delta = addr - lo.
// The arrays and work vectors carry at least 16 bytes of slack after their ends.
__device__ __forceinline__ void span16(const void *addr, size_t n, const char *&lo,
                                       uint32_t &delta, uint32_t &bytes) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(addr);
  lo = reinterpret_cast<const char *>(a & ~(uintptr_t) 15);
  delta = (uint32_t) (a & 15u);
  bytes = (uint32_t) ((delta + n + 15) & ~(size_t) 15);
}

// complex panel entries: nearfield and coupling panels of a complex operator
__device__ __forceinline__ bool complex_panel(uint32_t kind) {
  return kind == H2B_MV_NEAR || kind == H2B_MV_COUPLING;
}

template <bool CX, typename T>
__device__ __forceinline__ const char *panel_addr(const MvLaunch &L, const MvItem &m, size_t &n) {
  const uint32_t kind = m.flags & H2B_MV_KIND;
  const size_t esz = sizeof(T) * ((CX && complex_panel(kind)) ? 2 : 1);
  n = (size_t) m.rows * m.cols * esz;
  return reinterpret_cast<const char *>(L.A[kind]) + m.p * esz;
}

// entry e of a panel (complex entries as one vector load: a complex panel starts on a multiple of
// its entry size, so the stage copy keeps that alignment)
template <bool PCX, typename T>
__device__ __forceinline__ void entry(const T *P, size_t e, double &re, double &im) {
  if constexpr (PCX) {
    using V2 = typename std::conditional<std::is_same<T, float>::value, float2, double2>::type;
    const V2 v = reinterpret_cast<const V2 *>(P)[e];
    re = (double) v.x;
    im = (double) v.y;
  } else {
    re = (double) P[e];
    im = 0.0;
  }
}

// The columns of a product that a warp multiplies a panel with at once: their x slices in the stage
// and their y slices.
template <int NQ>
struct Cols {
  const double *x[NQ];
  double *y[NQ];
  int n;
};

// y_q[0, R) += P x_q[0, C) by one warp for the n <= NQ columns q: lanes take rows (SL slots of 32), the
// warp runs over the panel's columns, each entry read once for all q; one atomic addition per row
// and column.
template <bool CX, bool PCX, typename T, int SL, int NQ>
__device__ __forceinline__ void warp_gemv_n(const T *__restrict__ P, uint32_t R, uint32_t C,
                                            const Cols<NQ> &v, uint32_t lane) {
  constexpr int W = CX ? 2 : 1;
  double sr[SL][NQ], si[SL][NQ];
  bool on[SL];
#pragma unroll
  for (int j = 0; j < SL; j++) {
    on[j] = lane + 32u * j < R;
#pragma unroll
    for (int q = 0; q < NQ; q++) sr[j][q] = si[j][q] = 0.0;
  }
#pragma unroll 4
  for (uint32_t c = 0; c < C; c++) {
    double xr[NQ], xi[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      xr[q] = v.x[q][W * c];
      xi[q] = CX ? v.x[q][W * c + 1] : 0.0;
    }
    const T *col = P + (size_t) (PCX ? 2 : 1) * c * R;
#pragma unroll
    for (int j = 0; j < SL; j++) {
      if (on[j]) {
        double pr, pi;
        entry<PCX>(col, lane + 32u * j, pr, pi);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          if (PCX) {
            sr[j][q] = fma(pr, xr[q], fma(-pi, xi[q], sr[j][q]));
            si[j][q] = fma(pr, xi[q], fma(pi, xr[q], si[j][q]));
          } else {
            sr[j][q] = fma(pr, xr[q], sr[j][q]);
            if (CX) si[j][q] = fma(pr, xi[q], si[j][q]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < SL; j++) {
    if (on[j]) {
      const uint32_t r = lane + 32u * j;
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        if (q >= v.n) break;
        atomicAdd(v.y[q] + W * r, sr[j][q]);
        if (CX) atomicAdd(v.y[q] + W * r + 1, si[j][q]);
      }
    }
  }
}

// y_q[0, C) += P^T x_q[0, R) by one warp for the n <= NQ columns q, 32 panel columns at a time.  With cw
// of them the lanes form G = 32 / cp groups (cp: cw rounded up to a power of two); a lane takes one
// panel column and its group's part of the rows, and the groups' sums are added by shuffles, so that a
// panel of few columns (8 for complex rank 125) keeps every lane busy.  Lanes of neighbouring
// columns read P an odd number of entries apart, which falls in distinct banks: R apart for odd R,
// R + 1 for even R (a lane starts its rows at its column's number and wraps around).
template <bool CX, bool PCX, typename T, int NQ>
__device__ __forceinline__ void warp_gemv_t(const T *__restrict__ P, uint32_t R, uint32_t C,
                                            const Cols<NQ> &v, uint32_t lane) {
  constexpr int W = CX ? 2 : 1;
  for (uint32_t c0 = 0; c0 < C; c0 += 32) {
    const uint32_t cw = min(32u, C - c0), cp = cw > 1 ? 1u << (32 - __clz(cw - 1)) : 1u;
    const uint32_t col = lane & (cp - 1u), G = 32u / cp, grp = lane / cp;
    const uint32_t r0 = grp * R / G, len = (grp + 1) * R / G - r0;
    const bool on = col < cw;
    double sr[NQ], si[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) sr[q] = si[q] = 0.0;
    if (on && len > 0) {
      const T *p = P + (size_t) (PCX ? 2 : 1) * ((size_t) (c0 + col) * R + r0);
      uint32_t r = (R & 1u) ? 0u : col % len;
#pragma unroll 4
      for (uint32_t it = 0; it < len; it++) {
        double pr, pi;
        entry<PCX>(p, r, pr, pi);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          const double *x = v.x[q] + W * (r0 + r);
          const double xr = x[0], xi = CX ? x[1] : 0.0;
          if (PCX) {
            sr[q] = fma(pr, xr, fma(-pi, xi, sr[q]));
            si[q] = fma(pr, xi, fma(pi, xr, si[q]));
          } else {
            sr[q] = fma(pr, xr, sr[q]);
            if (CX) si[q] = fma(pr, xi, si[q]);
          }
        }
        r = r + 1 == len ? 0u : r + 1;
      }
    }
    for (uint32_t o = cp; o < 32u; o <<= 1) {
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        sr[q] += __shfl_xor_sync(0xffffffffu, sr[q], o);
        if (CX) si[q] += __shfl_xor_sync(0xffffffffu, si[q], o);
      }
    }
    if (on && grp == 0) {
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        if (q >= v.n) break;
        atomicAdd(v.y[q] + W * (c0 + col), sr[q]);
        if (CX) atomicAdd(v.y[q] + W * (c0 + col) + 1, si[q]);
      }
    }
  }
}

template <bool CX, bool PCX, typename T, int NQ>
__device__ __forceinline__ void gemv_n_any(const T *P, uint32_t R, uint32_t C, const Cols<NQ> &v,
                                           uint32_t lane) {
  switch ((R + 31) >> 5) {
    case 1: warp_gemv_n<CX, PCX, T, 1, NQ>(P, R, C, v, lane); break;
    case 2: warp_gemv_n<CX, PCX, T, 2, NQ>(P, R, C, v, lane); break;
    case 3: warp_gemv_n<CX, PCX, T, 3, NQ>(P, R, C, v, lane); break;
    default: warp_gemv_n<CX, PCX, T, 4, NQ>(P, R, C, v, lane); break;
  }
}

// Warp nw produces: for each of the CTA's items i (list entry first + blockIdx.x + i gridDim.x)
// it copies the panel and the x slice of every right-hand side into stage i % S (one bulk copy
// each, completion on full[s]) once the stage's previous item has been released (empty[s]), and
// puts the descriptor in the stage's slot.
// Consumer warp w multiplies the items i = w, w + nw, ... alone: S is a multiple of nw, so stage
// i % S always belongs to the same warp, and no barrier joins the consumer warps.  Every wait is
// bounded; a warp whose wait runs out sets the error flag and leaves, and the others' bounded
// waits end the CTA.
// NQ: columns multiplied per read of a panel from the stage (1, or MULTI for several columns).
template <bool CX, typename T, int NQ>
__global__ void __launch_bounds__(MAXTHREADS) mv_items_kernel(MvLaunch L) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int W = CX ? 2 : 1;
  const uint32_t S = L.stages;
  unsigned char *stage0 = smem;
  MvItem *slot = reinterpret_cast<MvItem *>(smem + (size_t) S * L.stage_bytes);
  uint64_t *full = reinterpret_cast<uint64_t *>(slot + S);
  uint64_t *empty = full + S;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t mine = L.n > blockIdx.x ? (L.n - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < S; s++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&full[s])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&empty[s])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == L.nw) {
    // ---- producer (one lane): the next descriptor is fetched while the current copies run
    if (lane != 0 || mine == 0) return;
    MvItem m = L.items[L.first + blockIdx.x];
    uint32_t i = 0;
    bool ok = true;
    for (; i < mine; i++) {
      const uint32_t s = i % S;
      if (i >= S && !(ok = bar_wait(smem_addr(&empty[s]), ((i / S) - 1) & 1u))) break;
      const uint32_t bar = smem_addr(&full[s]);
      slot[s] = m;
      size_t n;
      const char *pa = panel_addr<CX, T>(L, m, n), *lo;
      uint32_t delta, bytes;
      span16(pa, n, lo, delta, bytes);
      const int t = m.flags & H2B_MV_KIND;
      const size_t xn = (size_t) W * sizeof(double) * ((m.flags & H2B_MV_TRANS) ? m.rows : m.cols);
      // only the columns whose system is still running are copied; an item with none (its
      // surface's systems have all stopped) loads nothing and its stage completes at once
      uint32_t total = 0;
      bool any = false;
      for (uint32_t q = 0; q < L.nrhs; q++) {
        if (!col_on(L.mask, L.nseg, m.seg, q)) continue;
        const char *xl;
        uint32_t xd, xb;
        span16(L.X[t] + q * L.sx[t] + (size_t) W * m.xo, xn, xl, xd, xb);
        total += xb;
        any = true;
      }
      if (!any) {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
      } else {
        total += bytes;
        const uint32_t dst = smem_addr(stage0 + (size_t) s * L.stage_bytes);
        // the generic-proxy reads of the stage's previous contents are ordered before these
        // copies
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(total)
                     : "memory");
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(dst), "l"(lo), "r"(bytes), "r"(bar)
            : "memory");
        for (uint32_t q = 0; q < L.nrhs; q++) {
          if (!col_on(L.mask, L.nseg, m.seg, q)) continue;
          const char *xl;
          uint32_t xd, xb;
          span16(L.X[t] + q * L.sx[t] + (size_t) W * m.xo, xn, xl, xd, xb);
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
              "[%3];" ::"r"(dst + L.panel_bytes + q * L.xcol_bytes), "l"(xl), "r"(xb), "r"(bar)
              : "memory");
        }
      }
      if (i + 1 < mine) m = L.items[L.first + blockIdx.x + (i + 1) * gridDim.x];
    }
    if (!ok) {
      // a wait ran out: flag it and wait (bounded) for the copies this warp issued before it
      // leaves the CTA's shared memory (the consumers give up at their next stage)
      atomicExch(L.err, 1);
      for (uint32_t j = i > S ? i - S : 0; j < i; j++)
        bar_wait(smem_addr(&full[j % S]), (j / S) & 1u);
    }
    return;
  }
  if (warp > L.nw) return;

  // ---- consumers
  for (uint32_t i = warp; i < mine; i += L.nw) {
    const uint32_t s = i % S;
    if (!bar_wait(smem_addr(&full[s]), (i / S) & 1u)) {
      if (lane == 0) atomicExch(L.err, 1);
      return;
    }
    const MvItem m = slot[s];
    const unsigned char *stage = stage0 + (size_t) s * L.stage_bytes;
    size_t n;
    const char *pa = panel_addr<CX, T>(L, m, n), *lo;
    uint32_t delta, bytes;
    span16(pa, n, lo, delta, bytes);
    const T *P = reinterpret_cast<const T *>(stage + delta);
    const int t = m.flags & H2B_MV_KIND;
    const bool trans = (m.flags & H2B_MV_TRANS) != 0;
    // the running columns, up to NQ at a time (unused places repeat the last one and write nothing)
    for (uint32_t q = 0; q < L.nrhs;) {
      Cols<NQ> v;
      uint32_t at[NQ];
      v.n = 0;
#pragma unroll
      for (int j = 0; j < NQ; j++) {
        while (q < L.nrhs && !col_on(L.mask, L.nseg, m.seg, q)) q++;
        if (q < L.nrhs && (NQ == 1 || (uint32_t) j < L.group)) {
          at[j] = q++;
          v.n = j + 1;
        } else {
          at[j] = j > 0 ? at[j - 1] : 0u;
        }
      }
      if (v.n == 0) break;
#pragma unroll
      for (int j = 0; j < NQ; j++) {
        const double *x = L.X[t] + at[j] * L.sx[t] + (size_t) W * m.xo;
        v.x[j] = reinterpret_cast<const double *>(stage + L.panel_bytes + at[j] * L.xcol_bytes +
                                                  (reinterpret_cast<uintptr_t>(x) & 15u));
        v.y[j] = L.Y[t] + at[j] * L.sy[t] + (size_t) W * m.yo;
      }
      if (trans) warp_gemv_t<CX, false, T, NQ>(P, m.rows, m.cols, v, lane);
      else if (CX && complex_panel(t)) gemv_n_any<CX, CX, T, NQ>(P, m.rows, m.cols, v, lane);
      else gemv_n_any<CX, false, T, NQ>(P, m.rows, m.cols, v, lane);
    }
    __syncwarp();
    if (lane == 0)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&empty[s]))
                   : "memory");
  }
}

// Coupling panels.  A warp takes a run of consecutive panels of one block (several runs per warp, a
// block's panels are neighbours in the list) through a stage of its own and keeps the block's row
// sums in registers (SL slots of 32 rows, NQ columns), so that they reach yt once per run and not once
// per panel: for complex rank 125 a 16 KiB panel has 8 columns, and adding its 125 rows per panel
// took 485M FP64 additions to L2 for a product of 49152 triangles with five columns.  A panel
// that stands for its block and the transposed one (H2B_MV_SYM) is multiplied a second time,
// transposed, with the row cluster's x, which comes with the first of a run's panels that takes it.  A
// warp issues its own copies (panel and x slices, completion on its mbarrier) as soon as it has read the
// panel before: the other warps of the SM cover the wait, and no warp waits for another's copy to be
// issued (one producer lane for four warps took twice as long on small matrices).  Waits are bounded;
// nrhs <= NQ.
// 49152 triangles, m = 5, complex: a product with five columns 9.6 ms as five products, 6.2 with the
// columns together and panels added one by one, 3.2 with this kernel.  32768 triangles, m = 4, real:
// 104 us reading every block, 88 reading one of two.
constexpr uint32_t CP_WARPS = 4;  // warps of a CTA
template <bool CX, typename T, int SL, int NQ>
__global__ void __launch_bounds__(CP_WARPS * 32) mv_coupling_kernel(MvLaunch L) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int W = CX ? 2 : 1;
  constexpr int t = H2B_MV_COUPLING;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  // the warp's stage (panel, x slices), row slices and barrier
  unsigned char *stage = smem + (size_t) warp * L.stage_bytes;
  double *x2 = reinterpret_cast<double *>(smem + (size_t) L.nw * L.stage_bytes) +
               (size_t) warp * L.nrhs * L.x2_doubles;
  const uint32_t bar = smem_addr(
      reinterpret_cast<uint64_t *>(smem + (size_t) L.nw * (L.stage_bytes + 8u * L.nrhs * L.x2_doubles)) + warp);
  if (lane == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  // the warp's runs: every wall-th
  const uint32_t nruns = (L.n + L.run - 1) / L.run, wall = gridDim.x * L.nw;
  // lane 0: copies panel m and its x slices; head: the row slices too, where it takes them
  auto issue = [&](const MvItem &m, bool head) {
    size_t n;
    const char *pa = panel_addr<CX, T>(L, m, n), *lo, *xl;
    uint32_t delta, bytes, total = 0, xd, xb;
    span16(pa, n, lo, delta, bytes);
    const bool rows2 = head && (m.flags & H2B_MV_SYM);
    const size_t xn = (size_t) W * sizeof(double) * m.cols, x2n = (size_t) W * sizeof(double) * m.rows;
    for (uint32_t q = 0; q < L.nrhs; q++) {
      if (!col_on(L.mask, L.nseg, m.seg, q)) continue;
      span16(L.X[t] + q * L.sx[t] + (size_t) W * m.xo, xn, xl, xd, xb);
      total += xb;
      if (rows2) {
        span16(L.X[t] + q * L.sx[t] + (size_t) W * m.yo, x2n, xl, xd, xb);
        total += xb;
      }
    }
    if (total == 0) {  // every column's system is done: nothing to copy
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
      return;
    }
    total += bytes;
    // the warp's reads of the stage are ordered before the copies into it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(total)
                 : "memory");
    auto copy = [&](uint32_t dst, const char *src, uint32_t nb) {
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
          "[%3];" ::"r"(dst), "l"(src), "r"(nb), "r"(bar)
          : "memory");
    };
    copy(smem_addr(stage), lo, bytes);
    for (uint32_t q = 0; q < L.nrhs; q++) {
      if (!col_on(L.mask, L.nseg, m.seg, q)) continue;
      span16(L.X[t] + q * L.sx[t] + (size_t) W * m.xo, xn, xl, xd, xb);
      copy(smem_addr(stage + L.panel_bytes + q * L.xcol_bytes), xl, xb);
      if (rows2) {
        span16(L.X[t] + q * L.sx[t] + (size_t) W * m.yo, x2n, xl, xd, xb);
        copy(smem_addr(x2 + (size_t) q * L.x2_doubles), xl, xb);
      }
    }
  };

  double sr[SL][NQ], si[SL][NQ];
  uint32_t at[NQ], ncol = 0, yo = UINT32_MAX, rows = 0;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    at[q] = 0;
#pragma unroll
    for (int j = 0; j < SL; j++) sr[j][q] = si[j][q] = 0.0;
  }
  auto flush = [&]() {
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      double *y = L.Y[t] + at[q] * L.sy[t] + (size_t) W * yo;
#pragma unroll
      for (int j = 0; j < SL; j++) {
        const uint32_t r = lane + 32u * j;
        if ((uint32_t) q < ncol && r < rows) {
          atomicAdd(y + W * r, sr[j][q]);
          if (CX) atomicAdd(y + W * r + 1, si[j][q]);
        }
        sr[j][q] = si[j][q] = 0.0;
      }
    }
  };
  uint32_t run = blockIdx.x * L.nw + warp, i = run * L.run, phase = 0;
  if (run >= nruns) return;
  MvItem m = L.items[L.first + i];
  if (lane == 0) issue(m, true);
  for (;;) {
    // the next panel's descriptor, on its way while this panel is multiplied
    uint32_t ni = i + 1;
    if (ni == min(L.n, (run + 1) * L.run)) {
      run += wall;
      ni = run < nruns ? run * L.run : L.n;
    }
    MvItem nm = m;
    if (ni < L.n) nm = L.items[L.first + ni];
    if (!bar_wait(bar, phase)) {
      // a wait ran out: flag it, wait once more (bounded) for the copies in flight, and leave
      if (lane == 0) atomicExch(L.err, 1);
      bar_wait(bar, phase);
      return;
    }
    phase ^= 1u;
    const bool sym = (m.flags & H2B_MV_SYM) != 0;
    if (m.yo != yo) {
      if (yo != UINT32_MAX) flush();
      yo = m.yo;
      rows = m.rows;
      // the running columns (unused places repeat the last one)
      ncol = 0;
      uint32_t q = 0;
#pragma unroll
      for (int u = 0; u < NQ; u++) {
        while (q < L.nrhs && !col_on(L.mask, L.nseg, m.seg, q)) q++;
        if (q < L.nrhs) {
          at[u] = q++;
          ncol = u + 1;
        } else {
          at[u] = u > 0 ? at[u - 1] : 0u;
        }
      }
    }
    if (ncol > 0) {
      size_t n;
      const char *pa = panel_addr<CX, T>(L, m, n);
      const T *P = reinterpret_cast<const T *>(stage + (reinterpret_cast<uintptr_t>(pa) & 15u));
      Cols<NQ> v;
      v.n = (int) ncol;
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        const double *x = L.X[t] + at[q] * L.sx[t] + (size_t) W * m.xo;
        v.x[q] = reinterpret_cast<const double *>(stage + L.panel_bytes + at[q] * L.xcol_bytes +
                                                  (reinterpret_cast<uintptr_t>(x) & 15u));
      }
      // enough columns in flight to cover the shared-memory latency
      constexpr int U = SL * NQ <= 4 ? 8 : SL * NQ <= 8 ? 4 : 2;
#pragma unroll U
      for (uint32_t c = 0; c < m.cols; c++) {
        double xr[NQ], xi[NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          xr[q] = v.x[q][W * c];
          xi[q] = CX ? v.x[q][W * c + 1] : 0.0;
        }
        const T *col = P + (size_t) W * c * rows;
#pragma unroll
        for (int u = 0; u < SL; u++) {
          if (lane + 32u * u < rows) {
            double pr, pi;
            entry<CX>(col, lane + 32u * u, pr, pi);
#pragma unroll
            for (int q = 0; q < NQ; q++) {
              if (CX) {
                sr[u][q] = fma(pr, xr[q], fma(-pi, xi[q], sr[u][q]));
                si[u][q] = fma(pr, xi[q], fma(pi, xr[q], si[u][q]));
              } else {
                sr[u][q] = fma(pr, xr[q], sr[u][q]);
              }
            }
          }
        }
      }
      if (sym) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
          const double *x = L.X[t] + at[q] * L.sx[t] + (size_t) W * yo;
          v.x[q] = reinterpret_cast<const double *>(
              reinterpret_cast<const unsigned char *>(x2 + at[q] * L.x2_doubles) +
              (reinterpret_cast<uintptr_t>(x) & 15u));
          v.y[q] = L.Y[t] + at[q] * L.sy[t] + (size_t) W * m.xo;
        }
        warp_gemv_t<CX, CX, T, NQ>(P, rows, m.cols, v, lane);
      }
    }
    __syncwarp();
    if (ni >= L.n) break;
    // the row slices are there already when the panel before, of the same run and row cluster, took
    // them; a panel without H2B_MV_SYM takes none (partitions that are not symmetric mix the two)
    if (lane == 0) issue(nm, nm.yo != m.yo || ni != i + 1 || !sym);
    m = nm;
    i = ni;
  }
  flush();
}

// Columns multiplied per read of a panel when a product has several: four complex columns of a
// 125-row panel are 32 sums per lane.
constexpr int MULTI = 4;

// Stage layout of launch g (0 forward + nearfield, 1 coupling, 2 backward): the panel (FP64 panel
// bytes scaled to the storage type, plus 32 bytes for the alignment and rounding slack) and the x
// slices of nrhs columns.
template <typename T>
uint32_t panel_region(const MvItems &ph, int g) {
  const size_t b = (size_t) ph.max_bytes[g] * sizeof(T) / sizeof(double) + 32;
  return (uint32_t) ((b + 127) & ~(size_t) 127);
}

template <bool CX>
uint32_t slice_region(uint32_t n) {
  return n ? (uint32_t) ((sizeof(double) * (CX ? 2 : 1) * n + 32 + 15) & ~(size_t) 15) : 0u;
}
template <bool CX>
uint32_t xcol_region(const MvItems &ph, int g) {
  return slice_region<CX>(ph.max_x[g]);
}

template <bool CX, typename T>
uint32_t stage_of(const MvItems &ph, int g, uint32_t nrhs) {
  const size_t b = panel_region<T>(ph, g) + (size_t) nrhs * xcol_region<CX>(ph, g);
  return (uint32_t) ((b + 127) & ~(size_t) 127);
}

template <bool CX, typename T>
size_t smem_of(const MvItems &ph, int g, uint32_t stages, uint32_t nrhs) {
  return (size_t) stages * (stage_of<CX, T>(ph, g, nrhs) + sizeof(MvItem) + 16);
}

// the largest of a product's launches
template <bool CX, typename T>
size_t smem_most(const MvItems &ph, uint32_t stages, uint32_t nrhs) {
  size_t b = 0;
  for (int g = 0; g < 3; g += 2) b = std::max(b, smem_of<CX, T>(ph, g, stages, nrhs));
  return b;
}

// consumer warps and ring stages of a launch shape (stages per consumer warp 1..4)
void ring_shape(const MvmPlan *p, uint32_t &nw, uint32_t &stages) {
  nw = (uint32_t) std::max(1, std::min(MAXTHREADS / 32 - 1, p->warps));
  stages = nw * (uint32_t) std::max(1, std::min(4, p->stages));
}

template <bool CX, typename T, int NQ>
int launch_items(const MvmPlan *p, const MvLaunch &L, size_t smem, cudaStream_t st) {
  const int threads = (int) (L.nw + 1) * 32;
  H2B_CUDA_TRY((h2b_allow_smem<mv_items_kernel<CX, T, NQ>>()));
  int occ = 0;
  H2B_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mv_items_kernel<CX, T, NQ>,
                                                             threads, smem));
  if (occ < 1) {
    h2b_set_error("matvec: the item kernel does not fit an SM (%zu bytes of shared memory)", smem);
    return H2B_ERR_ARG;
  }
  const int sms = p->num_sms > 0 ? p->num_sms : 148;
  const int per_sm = std::min(occ, std::max(1, p->ctas_per_sm));
  const uint32_t grid = std::min<uint32_t>(L.n, (uint32_t) (per_sm * sms));
  mv_items_kernel<CX, T, NQ><<<grid, threads, smem, st>>>(L);
  h2b_note_launch();
  return H2B_OK;
}

// The items [first, last) of one launch's kinds (g: 0 forward + nearfield, 2 backward).
template <bool CX, typename T>
int launch_range(const MvmPlan *p, const MvItems &ph, const MvLaunch &base, uint32_t first,
                 uint32_t last, cudaStream_t st) {
  if (last <= first) return H2B_OK;
  const int g = first >= ph.start[H2B_MV_BACKWARD] ? 2 : 0;
  MvLaunch L = base;
  L.items = ph.items;
  L.first = first;
  L.n = last - first;
  ring_shape(p, L.nw, L.stages);
  L.panel_bytes = panel_region<T>(ph, g);
  L.xcol_bytes = xcol_region<CX>(ph, g);
  L.stage_bytes = stage_of<CX, T>(ph, g, L.nrhs);
  const uint32_t groups = (L.nrhs + MULTI - 1) / MULTI;
  L.group = (L.nrhs + groups - 1) / groups;
  const size_t smem = smem_of<CX, T>(ph, g, L.stages, L.nrhs);
  if (smem > H2B_MAX_DYN_SMEM || ph.max_rows > MAXROWS || ph.max_x[g] > 65536) {
    h2b_set_error("matvec: item panel of %u bytes / %u rows / %u right-hand sides exceeds the "
                  "kernel's limits (%zu bytes of shared memory)",
                  ph.max_bytes[g], ph.max_rows, L.nrhs, smem);
    return H2B_ERR_ARG;
  }
  return L.nrhs > 1 ? launch_items<CX, T, MULTI>(p, L, smem, st)
                    : launch_items<CX, T, 1>(p, L, smem, st);
}

// Shared memory of the coupling kernel for n columns.
template <bool CX, typename T>
size_t coupling_smem(const MvItems &ph, uint32_t nw, uint32_t n) {
  const size_t x2 = slice_region<CX>(ph.max_x2[1]);
  return (size_t) nw * (stage_of<CX, T>(ph, 1, n) + n * x2 + 8);
}

template <bool CX, typename T, int SL, int NQ>
int launch_coupling_of(const MvmPlan *p, const MvItems &ph, MvLaunch &L, cudaStream_t st) {
  const size_t smem = coupling_smem<CX, T>(ph, L.nw, L.nrhs);
  const int threads = (int) L.nw * 32;
  H2B_CUDA_TRY((h2b_allow_smem<mv_coupling_kernel<CX, T, SL, NQ>>()));
  int occ = 0;
  H2B_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      &occ, mv_coupling_kernel<CX, T, SL, NQ>, threads, smem));
  if (smem > H2B_MAX_DYN_SMEM || occ < 1) {
    h2b_set_error("matvec: the coupling kernel does not fit an SM (%zu bytes of shared memory)", smem);
    return H2B_ERR_ARG;
  }
  const int sms = p->num_sms > 0 ? p->num_sms : 148;
  // runs: at least six per warp, so that the last round is short, at most a block each
  const uint32_t all = (uint32_t) (occ * sms) * L.nw;
  L.run = std::max(1u, std::min(ph.per_block, L.n / (6u * all)));
  const uint32_t runs = (L.n + L.run - 1) / L.run;
  const uint32_t grid = std::min<uint32_t>((runs + L.nw - 1) / L.nw, (uint32_t) (occ * sms));
  mv_coupling_kernel<CX, T, SL, NQ><<<grid, threads, smem, st>>>(L);
  h2b_note_launch();
  return H2B_OK;
}

// Columns of one coupling launch.
constexpr uint32_t CP_MAX = 5;

template <bool CX, typename T, int SL>
int launch_coupling_n(const MvmPlan *p, const MvItems &ph, MvLaunch &L, cudaStream_t st) {
  if (L.nrhs == 1) return launch_coupling_of<CX, T, SL, 1>(p, ph, L, st);
  if (L.nrhs <= 4) return launch_coupling_of<CX, T, SL, 4>(p, ph, L, st);
  return launch_coupling_of<CX, T, SL, (int) CP_MAX>(p, ph, L, st);
}

// The coupling items, up to CP_MAX columns per launch (balanced).  Consumer warps: the shape that
// keeps the most warps on an SM with at least one stage each.
template <bool CX, typename T>
int launch_coupling(const MvmPlan *p, const MvItems &ph, const MvLaunch &base, cudaStream_t st) {
  const uint32_t first = ph.start[H2B_MV_COUPLING], last = ph.start[H2B_MV_BACKWARD];
  if (last <= first) return H2B_OK;
  const uint32_t groups = (base.nrhs + CP_MAX - 1) / CP_MAX, per = (base.nrhs + groups - 1) / groups;
  for (uint32_t q0 = 0; q0 < base.nrhs; q0 += per) {
    MvLaunch L = base;
    L.items = ph.items;
    L.first = first;
    L.n = last - first;
    L.nrhs = std::min(per, base.nrhs - q0);
    L.X[H2B_MV_COUPLING] += q0 * L.sx[H2B_MV_COUPLING];
    L.Y[H2B_MV_COUPLING] += q0 * L.sy[H2B_MV_COUPLING];
    if (L.mask) L.mask += (size_t) q0 * L.nseg;
    L.nw = CP_WARPS;
    while (L.nw > 1 && coupling_smem<CX, T>(ph, L.nw, L.nrhs) > 110u * 1024u) L.nw--;
    L.panel_bytes = panel_region<T>(ph, 1);
    L.xcol_bytes = xcol_region<CX>(ph, 1);
    L.stage_bytes = stage_of<CX, T>(ph, 1, L.nrhs);
    L.x2_doubles = slice_region<CX>(ph.max_x2[1]) / 8u;
    if (p->k > MAXROWS) {
      h2b_set_error("matvec: rank %d exceeds %d", p->k, MAXROWS);
      return H2B_ERR_ARG;
    }
    const int rc = p->k <= 32   ? launch_coupling_n<CX, T, 1>(p, ph, L, st)
                   : p->k <= 64 ? launch_coupling_n<CX, T, 2>(p, ph, L, st)
                                : launch_coupling_n<CX, T, 4>(p, ph, L, st);
    if (rc != H2B_OK) return rc;
  }
  return H2B_OK;
}

template <bool CX, bool SINGLE>
int launch_all(const MvmPlan *p, const double *x, size_t ldx, double *y, size_t ldy, double ar,
               double ai, const MvmVecs &v, cudaStream_t st) {
  using T = typename std::conditional<SINGLE, float, double>::type;
  const size_t W = CX ? 2 : 1;
  const int sms = p->num_sms > 0 ? p->num_sms : 148;
  const uint32_t zn = p->nrow > p->ncol ? p->nrow : p->ncol;
  const uint32_t gz = std::min<uint32_t>((zn + 255) / 256 + 1, (uint32_t) (4 * sms));
  const size_t nyp = W * p->nrow, nxt = W * (size_t) p->k * p->ncol_clusters,
               nyt = W * (size_t) p->k * p->nrow_clusters;
  gather_zero_kernel<CX><<<gz, 256, 0, st>>>(x, ldx, p->cidx, p->ncol, v, nyp, nxt, nyt);
  h2b_note_launch();
  MvLaunch L{};
  L.nrhs = v.nrhs;
  L.nseg = v.nseg;
  L.mask = v.mask;
  L.err = p->err;
  L.A[H2B_MV_FORWARD] = SINGLE ? (const void *) p->fWc : (const void *) p->Wc;
  L.A[H2B_MV_NEAR] = SINGLE ? (const void *) p->fN : (const void *) p->N;
  L.A[H2B_MV_COUPLING] = SINGLE ? (const void *) p->fS : (const void *) p->S;
  L.A[H2B_MV_BACKWARD] = SINGLE ? (const void *) p->fWr : (const void *) p->Wr;
  L.X[H2B_MV_FORWARD] = v.xp, L.Y[H2B_MV_FORWARD] = v.xt;
  L.sx[H2B_MV_FORWARD] = v.sxp, L.sy[H2B_MV_FORWARD] = v.sxt;
  L.X[H2B_MV_NEAR] = v.xp, L.Y[H2B_MV_NEAR] = v.yp;
  L.sx[H2B_MV_NEAR] = v.sxp, L.sy[H2B_MV_NEAR] = v.syp;
  L.X[H2B_MV_COUPLING] = v.xt, L.Y[H2B_MV_COUPLING] = v.yt;
  L.sx[H2B_MV_COUPLING] = v.sxt, L.sy[H2B_MV_COUPLING] = v.syt;
  L.X[H2B_MV_BACKWARD] = v.yt, L.Y[H2B_MV_BACKWARD] = v.yp;
  L.sx[H2B_MV_BACKWARD] = v.syt, L.sy[H2B_MV_BACKWARD] = v.syp;
  const MvItems &it = SINGLE ? p->items_single : p->items;
  // forward + nearfield, coupling (reads xt), backward (reads yt)
  int rc = launch_range<CX, T>(p, it, L, 0, it.start[H2B_MV_COUPLING], st);
  if (rc == H2B_OK) rc = launch_coupling<CX, T>(p, it, L, st);
  if (rc == H2B_OK) rc = launch_range<CX, T>(p, it, L, it.start[H2B_MV_BACKWARD], it.n, st);
  if (rc != H2B_OK) return rc;
  scatter_multi_kernel<CX><<<gz, 256, 0, st>>>(v, p->ridx, y, ldy, p->nrow, ar, ai);
  h2b_note_launch();
  H2B_CUDA_TRY(cudaGetLastError());
  return H2B_OK;
}

// The plan's own work vectors (one column, no mask).
MvmVecs plan_vecs(const MvmPlan *p) {
  MvmVecs v;
  v.xp = p->xp;
  v.yp = p->yp;
  v.xt = p->xt;
  v.yt = p->yt;
  v.sxp = v.syp = v.sxt = v.syt = 0;
  v.nrhs = 1;
  v.nseg = 1;
  v.mask = nullptr;
  return v;
}

bool has_single(const MvmPlan *p) { return p->fWc && p->fWr && p->fN && p->fS; }

// xs = b xp and xp = a xp, n entries (complex: interleaved pairs).
template <bool CX>
__global__ void scale_copy_kernel(double *__restrict__ xp, double *__restrict__ xs, uint32_t n,
                                  double ar, double ai, double br, double bi) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (CX) {
      const double re = xp[2 * i], im = xp[2 * i + 1];
      xs[2 * i] = br * re - bi * im;
      xs[2 * i + 1] = br * im + bi * re;
      xp[2 * i] = ar * re - ai * im;
      xp[2 * i + 1] = ar * im + ai * re;
    } else {
      const double v = xp[i];
      xs[i] = br * v;
      xp[i] = ar * v;
    }
  }
}

// y += a A x + b B x for two matrices on one structure whose coupling matrices and row bases
// are equal (the caller checks): the forward transforms and nearfield blocks of both run on
// their own scaled copies of x into p's accumulators, then p's coupling matrices and row basis
// are applied once.
template <bool CX, bool SINGLE>
int launch_pair(const MvmPlan *p, const MvmPlan *q, const double *x, double *y, double ar,
                double ai, double br, double bi, const MvmVecs &v, double *xq, cudaStream_t st) {
  using T = typename std::conditional<SINGLE, float, double>::type;
  const size_t W = CX ? 2 : 1;
  const int sms = p->num_sms > 0 ? p->num_sms : 148;
  const uint32_t zn = p->nrow > p->ncol ? p->nrow : p->ncol;
  const uint32_t gz = std::min<uint32_t>((zn + 255) / 256 + 1, (uint32_t) (4 * sms));
  const size_t nyp = W * p->nrow, nxt = W * (size_t) p->k * p->ncol_clusters,
               nyt = W * (size_t) p->k * p->nrow_clusters;
  gather_zero_kernel<CX><<<gz, 256, 0, st>>>(x, 0, p->cidx, p->ncol, v, nyp, nxt, nyt);
  h2b_note_launch();
  scale_copy_kernel<CX><<<gz, 256, 0, st>>>(v.xp, xq, p->ncol, ar, ai, br, bi);
  h2b_note_launch();
  MvLaunch L{};
  L.nrhs = 1;
  L.nseg = 1;
  L.mask = nullptr;
  L.err = p->err;
  L.A[H2B_MV_FORWARD] = SINGLE ? (const void *) p->fWc : (const void *) p->Wc;
  L.A[H2B_MV_NEAR] = SINGLE ? (const void *) p->fN : (const void *) p->N;
  L.A[H2B_MV_COUPLING] = SINGLE ? (const void *) p->fS : (const void *) p->S;
  L.A[H2B_MV_BACKWARD] = SINGLE ? (const void *) p->fWr : (const void *) p->Wr;
  L.X[H2B_MV_FORWARD] = v.xp, L.Y[H2B_MV_FORWARD] = v.xt;
  L.X[H2B_MV_NEAR] = v.xp, L.Y[H2B_MV_NEAR] = v.yp;
  L.X[H2B_MV_COUPLING] = v.xt, L.Y[H2B_MV_COUPLING] = v.yt;
  L.X[H2B_MV_BACKWARD] = v.yt, L.Y[H2B_MV_BACKWARD] = v.yp;
  MvLaunch Lq = L;
  Lq.A[H2B_MV_FORWARD] = SINGLE ? (const void *) q->fWc : (const void *) q->Wc;
  Lq.A[H2B_MV_NEAR] = SINGLE ? (const void *) q->fN : (const void *) q->N;
  Lq.X[H2B_MV_FORWARD] = xq;
  Lq.X[H2B_MV_NEAR] = xq;
  const MvItems &it = SINGLE ? p->items_single : p->items;
  const MvItems &iq = SINGLE ? q->items_single : q->items;
  int rc = launch_range<CX, T>(p, it, L, 0, it.start[H2B_MV_COUPLING], st);
  if (rc == H2B_OK) rc = launch_range<CX, T>(p, iq, Lq, 0, iq.start[H2B_MV_COUPLING], st);
  if (rc == H2B_OK) rc = launch_coupling<CX, T>(p, it, L, st);
  if (rc == H2B_OK) rc = launch_range<CX, T>(p, it, L, it.start[H2B_MV_BACKWARD], it.n, st);
  if (rc != H2B_OK) return rc;
  scatter_multi_kernel<CX><<<gz, 256, 0, st>>>(v, p->ridx, y, 0, p->nrow, 1.0, 0.0);
  h2b_note_launch();
  H2B_CUDA_TRY(cudaGetLastError());
  return H2B_OK;
}


}  // namespace

// The kernels that products of a plan launch with entries of type T: one kernel's rank class of the
// coupling's three, every number of columns.
template <bool CX, typename T, int SL>
static int prepare_coupling(void) {
  H2B_CUDA_TRY((h2b_allow_smem<mv_coupling_kernel<CX, T, SL, 1>>()));
  H2B_CUDA_TRY((h2b_allow_smem<mv_coupling_kernel<CX, T, SL, 4>>()));
  H2B_CUDA_TRY((h2b_allow_smem<mv_coupling_kernel<CX, T, SL, (int) CP_MAX>>()));
  return H2B_OK;
}
template <bool CX, typename T>
static int prepare_type(int k) {
  H2B_CUDA_TRY((h2b_allow_smem<mv_items_kernel<CX, T, 1>>()));
  H2B_CUDA_TRY((h2b_allow_smem<mv_items_kernel<CX, T, MULTI>>()));
  return k <= 32 ? prepare_coupling<CX, T, 1>()
                 : k <= 64 ? prepare_coupling<CX, T, 2>() : prepare_coupling<CX, T, 4>();
}

extern "C" int h2b_mvm_prepare(const MvmPlan *p) {
  int rc = p->cx ? prepare_type<true, double>(p->k) : prepare_type<false, double>(p->k);
  if (rc == H2B_OK && p->fS)
    rc = p->cx ? prepare_type<true, float>(p->k) : prepare_type<false, float>(p->k);
  return rc;
}

static size_t smem_any(const MvmPlan *p, int single, uint32_t nrhs) {
  const MvItems &ph = single ? p->items_single : p->items;
  uint32_t nw, stages;
  ring_shape(p, nw, stages);
  if (p->cx)
    return single ? smem_most<true, float>(ph, stages, nrhs) : smem_most<true, double>(ph, stages, nrhs);
  return single ? smem_most<false, float>(ph, stages, nrhs)
                : smem_most<false, double>(ph, stages, nrhs);
}

extern "C" size_t h2b_mvm_smem_bytes(const MvmPlan *p, int single) { return smem_any(p, single, 1); }

extern "C" uint32_t h2b_mvm_max_columns(const MvmPlan *p, int single) {
  // two groups of MULTI columns; fewer when their slices would leave an SM one CTA only
  uint32_t n = 2 * MULTI;
  while (n > 1 && smem_any(p, single, n) > H2B_MAX_DYN_SMEM / 2) n--;
  return n;
}

extern "C" int h2b_mvm_launch_single(const MvmPlan *p, const double *x, double *y, double ar,
                                     double ai, cudaStream_t st) {
  if (!has_single(p)) {
    h2b_set_error("matvec: no FP32 copy of the H2 matrix (h2b_h2matrix_make_single)");
    return H2B_ERR_ARG;
  }
  const MvmVecs v = plan_vecs(p);
  return p->cx ? launch_all<true, true>(p, x, 0, y, 0, ar, ai, v, st)
               : launch_all<false, true>(p, x, 0, y, 0, ar, ai, v, st);
}

extern "C" int h2b_mvm_launch(const MvmPlan *p, const double *x, double *y, double ar, double ai,
                              cudaStream_t st) {
  const MvmVecs v = plan_vecs(p);
  return p->cx ? launch_all<true, false>(p, x, 0, y, 0, ar, ai, v, st)
               : launch_all<false, false>(p, x, 0, y, 0, ar, ai, v, st);
}

extern "C" size_t h2b_mvm_pair_work_doubles(const MvmPlan *p) {
  // one column of p's vectors, then the second scaled copy of x with its own slack
  return h2b_mvm_work_doubles(p, 1) + (size_t) (p->cx ? 2 : 1) * p->ncol + 8;
}

extern "C" int h2b_mvm_launch_pair(const MvmPlan *p, const MvmPlan *q, int single,
                                   const double *x, double *y, double ar, double ai, double br,
                                   double bi, double *work, cudaStream_t st) {
  if (single && (!has_single(p) || !has_single(q))) {
    h2b_set_error("matvec: no FP32 copy of the H2 matrix (h2b_h2matrix_make_single)");
    return H2B_ERR_ARG;
  }
  MvmVecs v = plan_vecs(p);
  double *xq = q->xp;
  if (work) {
    const size_t W = p->cx ? 2 : 1;
    v.xp = work;
    v.yp = v.xp + W * p->ncol;
    v.xt = v.yp + W * p->nrow;
    v.yt = v.xt + W * (size_t) p->k * p->ncol_clusters;
    xq = work + h2b_mvm_work_doubles(p, 1);
  }
  if (p->cx)
    return single ? launch_pair<true, true>(p, q, x, y, ar, ai, br, bi, v, xq, st)
                  : launch_pair<true, false>(p, q, x, y, ar, ai, br, bi, v, xq, st);
  return single ? launch_pair<false, true>(p, q, x, y, ar, ai, br, bi, v, xq, st)
                : launch_pair<false, false>(p, q, x, y, ar, ai, br, bi, v, xq, st);
}

extern "C" size_t h2b_mvm_work_doubles(const MvmPlan *p, uint32_t nrhs) {
  const size_t W = p->cx ? 2 : 1;
  // the vectors and 8 doubles of slack after the last one (x slices are copied in 16-byte
  // aligned spans)
  return nrhs * W * ((size_t) p->ncol + p->nrow +
                     (size_t) p->k * (p->ncol_clusters + p->nrow_clusters)) + 8;
}

extern "C" int h2b_mvm_launch_batch(const MvmPlan *p, int single, uint32_t nrhs, const double *x,
                                    size_t ldx, double *y, size_t ldy, double ar, double ai,
                                    double *work, const uint32_t *mask, uint32_t nseg,
                                    cudaStream_t st) {
  if (single && !has_single(p)) {
    h2b_set_error("batched matvec: needs the FP32 copies (h2b_h2matrix_make_single)");
    return H2B_ERR_ARG;
  }
  if (nrhs == 0) {
    h2b_set_error("batched matvec: no columns");
    return H2B_ERR_ARG;
  }
  const size_t W = p->cx ? 2 : 1;
  MvmVecs v;
  v.sxp = W * p->ncol;
  v.syp = W * p->nrow;
  v.sxt = W * (size_t) p->k * p->ncol_clusters;
  v.syt = W * (size_t) p->k * p->nrow_clusters;
  v.xp = work;
  v.yp = v.xp + nrhs * v.sxp;
  v.xt = v.yp + nrhs * v.syp;
  v.yt = v.xt + nrhs * v.sxt;
  v.nrhs = nrhs;
  v.nseg = nseg;
  v.mask = mask;
  if (p->cx)
    return single ? launch_all<true, true>(p, x, ldx, y, ldy, ar, ai, v, st)
                  : launch_all<true, false>(p, x, ldx, y, ldy, ar, ai, v, st);
  return single ? launch_all<false, true>(p, x, ldx, y, ldy, ar, ai, v, st)
                : launch_all<false, false>(p, x, ldx, y, ldy, ar, ai, v, st);
}
