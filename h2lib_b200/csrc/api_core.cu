// C-ABI implementation: status, device init, surfaces, operators and nearfield entry points.
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "api_internal.h"

// ------------------------------------------------------------------------------------------
// Status
// ------------------------------------------------------------------------------------------

static thread_local char g_err[1024] = "";

extern "C" void h2b_set_error(const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

extern "C" const char *h2b_last_error(void) { return g_err; }

extern "C" const char *h2b_version(void) { return "h2b200 0.1 (sm_100a)"; }

// Device whose constant tables are loaded; written under g_init_mutex (handles may be created
// from several host threads, e.g. the workers of a solve server).
static std::atomic<int> g_inited_device{-1};
static std::mutex g_init_mutex;

extern "C" int h2b_device_init(int device) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    cudaGetLastError();
    h2b_set_error("no CUDA device available");
    return H2B_ERR_CUDA;
  }
  if (device < 0 || device >= n) {
    h2b_set_error("device %d out of range (%d devices)", device, n);
    return H2B_ERR_ARG;
  }
  H2B_CUDA_TRY(cudaSetDevice(device));
  int major = 0, minor = 0;
  H2B_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
  H2B_CUDA_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
  if (major != 10) {
    h2b_set_error("device %d is sm_%d%d; this library is built for sm_100a only", device,
                  major, minor);
    return H2B_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_init_mutex);
  if (g_inited_device != device) {
    int rc = h2b_near_upload_dist_rules();
    if (rc != H2B_OK) return rc;
    // keep freed stream-ordered memory in the device pool for reuse by later handles
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
      uint64_t keep = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
      // never make one handle's stream wait for another's to reuse a freed block
      int no = 0;
      cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no);
    }
    cudaGetLastError();
    g_inited_device = device;
  }
  return H2B_OK;
}

int h2b_ensure_device(void) {
  int dev = 0;
  if (g_inited_device >= 0) {
    H2B_CUDA_TRY(cudaGetDevice(&dev));
    if (dev == g_inited_device) return H2B_OK;
  } else if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    dev = 0;
  }
  return h2b_device_init(dev);
}

static std::atomic<unsigned long long> g_launches{0};

void h2b_note_launch(void) { g_launches.fetch_add(1, std::memory_order_relaxed); }

extern "C" int h2b_launch_count(uint64_t *n) {
  if (!n) return H2B_ERR_ARG;
  *n = g_launches.load(std::memory_order_relaxed);
  return H2B_OK;
}

extern "C" int h2b_device_memory(uint64_t out[4]) {
  if (!out) return H2B_ERR_ARG;
  int dev = 0;
  size_t fr = 0, tot = 0;
  H2B_CUDA_TRY(cudaGetDevice(&dev));
  H2B_CUDA_TRY(cudaMemGetInfo(&fr, &tot));
  cudaMemPool_t pool;
  uint64_t used = 0, reserved = 0;
  H2B_CUDA_TRY(cudaDeviceGetDefaultMemPool(&pool, dev));
  H2B_CUDA_TRY(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
  H2B_CUDA_TRY(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved));
  out[0] = fr;
  out[1] = tot;
  out[2] = used;
  out[3] = reserved;
  return H2B_OK;
}

bool h2b_is_device_ptr(const void *p) {
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

// ------------------------------------------------------------------------------------------
// Surfaces
// ------------------------------------------------------------------------------------------

extern "C" h2b_surface *h2b_surface_new(uint32_t vertices, const double *x, uint32_t triangles,
                                        const uint32_t *t, const double *n, const double *g) {
  if (!x || !t || !n || !g || vertices == 0 || triangles == 0) {
    h2b_set_error("h2b_surface_new: empty mesh or NULL array");
    return NULL;
  }
  for (uint64_t i = 0; i < 3ull * triangles; i++)
    if (t[i] >= vertices) {
      h2b_set_error("h2b_surface_new: triangle %llu references vertex %u >= %u",
                    (unsigned long long) (i / 3), t[i], vertices);
      return NULL;
    }
  if (h2b_ensure_device() != H2B_OK) return NULL;
  h2b_surface *s = new h2b_surface();
  s->nv = vertices;
  s->nt = triangles;
  s->x.assign(x, x + 3ull * vertices);
  s->t.assign(t, t + 3ull * triangles);
  s->n.assign(n, n + 3ull * triangles);
  s->g.assign(g, g + triangles);
  if (h2b_adjacency_build(vertices, triangles, s->t.data(), &s->adj) != H2B_OK) {
    delete s;
    h2b_set_error("h2b_surface_new: out of host memory");
    return NULL;
  }
  std::vector<TriRec> rec(triangles);
  for (uint32_t i = 0; i < triangles; i++) {
    TriRec &r = rec[i];
    memset(&r, 0, sizeof(r));
    const uint32_t *ti = t + 3ull * i;
    for (int d = 0; d < 3; d++) {
      r.a[d] = x[3ull * ti[0] + d];
      r.b[d] = x[3ull * ti[1] + d];
      r.c[d] = x[3ull * ti[2] + d];
      r.n[d] = n[3ull * i + d];
      r.v[d] = ti[d];
    }
    r.g = g[i];
  }
  // (an attribute query, not cudaGetDeviceProperties, which costs milliseconds per call)
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMallocAsync(&s->d_tri, sizeof(TriRec) * triangles, s->stream) != cudaSuccess ||
      cudaMallocAsync(&s->d_x, sizeof(double) * 3ull * vertices, s->stream) != cudaSuccess ||
      cudaMemcpyAsync(s->d_tri, rec.data(), sizeof(TriRec) * triangles, cudaMemcpyHostToDevice,
                      s->stream) != cudaSuccess ||
      cudaMemcpyAsync(s->d_x, x, sizeof(double) * 3ull * vertices, cudaMemcpyHostToDevice,
                      s->stream) != cudaSuccess ||
      cudaMallocAsync(&s->d_qrec, sizeof(QuadRec) * (size_t) triangles, s->stream) != cudaSuccess ||
      h2b_near_quad_records(s->d_tri, triangles, s->d_qrec, s->stream) != H2B_OK ||
      cudaMallocAsync(&s->d_vt_off, sizeof(uint32_t) * (vertices + 1ull), s->stream) != cudaSuccess ||
      cudaMallocAsync(&s->d_vt_tri, sizeof(uint32_t) * 3ull * triangles, s->stream) != cudaSuccess ||
      cudaMemcpyAsync(s->d_vt_off, s->adj.off, sizeof(uint32_t) * (vertices + 1ull),
                      cudaMemcpyHostToDevice, s->stream) != cudaSuccess ||
      cudaMemcpyAsync(s->d_vt_tri, s->adj.tri, sizeof(uint32_t) * 3ull * triangles,
                      cudaMemcpyHostToDevice, s->stream) != cudaSuccess ||
      cudaStreamSynchronize(s->stream) != cudaSuccess) {  // rec is read
    h2b_set_error("h2b_surface_new: %s", cudaGetErrorString(cudaGetLastError()));
    h2b_surface_del(s);
    return NULL;
  }
  s->device = dev;
  s->num_sms = sms;
  // neighbour lists: about 18 per triangle on usual meshes
  uint64_t room = 0;
  for (uint32_t v = 0; v < vertices; v++) {
    const uint64_t d = s->adj.off[v + 1] - s->adj.off[v];
    room += d * d;
  }
  if (room <= 64ull * triangles && room < UINT32_MAX) {
    uint32_t *cursor = nullptr;
    const cudaStream_t st = s->stream;
    if (cudaMallocAsync(&cursor, sizeof(uint32_t), st) != cudaSuccess ||
        cudaMallocAsync(&s->d_nb_off, sizeof(uint32_t) * (size_t) triangles, st) != cudaSuccess ||
        cudaMallocAsync(&s->d_nb_len, sizeof(uint32_t) * (size_t) triangles, st) != cudaSuccess ||
        cudaMallocAsync(&s->d_nb, sizeof(uint2) * room, st) != cudaSuccess ||
        cudaMemsetAsync(cursor, 0, sizeof(uint32_t), st) != cudaSuccess ||
        h2b_near_neighbours(s->d_tri, triangles, s->d_vt_off, s->d_vt_tri, cursor, s->d_nb_off,
                            s->d_nb_len, s->d_nb, st) != H2B_OK ||
        cudaFreeAsync(cursor, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
      h2b_set_error("h2b_surface_new: %s", cudaGetErrorString(cudaGetLastError()));
      h2b_surface_del(s);
      return NULL;
    }
  }
  return s;
}

extern "C" void h2b_surface_del(h2b_surface *s) {
  if (!s) return;
  // every entry point ends synchronised, so no kernel still reads these arrays; stream-ordered
  // frees do not synchronise the device (other handles keep running)
  if (s->d_tri) cudaFreeAsync(s->d_tri, s->stream);
  if (s->d_qrec) cudaFreeAsync(s->d_qrec, s->stream);
  if (s->d_x) cudaFreeAsync(s->d_x, s->stream);
  if (s->d_nb_off) cudaFreeAsync(s->d_nb_off, s->stream);
  if (s->d_nb_len) cudaFreeAsync(s->d_nb_len, s->stream);
  if (s->d_nb) cudaFreeAsync(s->d_nb, s->stream);
  if (s->d_vt_off) cudaFreeAsync(s->d_vt_off, s->stream);
  if (s->d_vt_tri) cudaFreeAsync(s->d_vt_tri, s->stream);
  if (s->stream) cudaStreamDestroy(s->stream);
  h2b_adjacency_free(&s->adj);
  delete s;
}

// ------------------------------------------------------------------------------------------
// Operators
// ------------------------------------------------------------------------------------------

extern "C" h2b_bem *h2b_bem_new(const h2b_surface *s, int pde, int layer, int row_basis,
                                int col_basis, uint32_t q_regular, uint32_t q_singular,
                                double k_re, double k_im, double alpha_re, double alpha_im) {
  if (!s) {
    h2b_set_error("h2b_bem_new: NULL surface");
    return NULL;
  }
  if ((pde != H2B_LAPLACE && pde != H2B_HELMHOLTZ) ||
      (layer != H2B_SLP && layer != H2B_DLP && layer != H2B_ADLP) ||
      (row_basis != H2B_BASIS_CONSTANT && row_basis != H2B_BASIS_LINEAR) ||
      (col_basis != H2B_BASIS_CONSTANT && col_basis != H2B_BASIS_LINEAR)) {
    h2b_set_error("h2b_bem_new: unknown pde/layer/basis (%d, %d, %d, %d)", pde, layer,
                  row_basis, col_basis);
    return NULL;
  }
  if (q_regular < 1 || q_regular > 5 || q_singular < 1 || q_singular > 8) {
    h2b_set_error("h2b_bem_new: quadrature orders (%u, %u) outside 1..5 / 1..8", q_regular,
                  q_singular);
    return NULL;
  }
  if (layer == H2B_SLP && (alpha_re != 0.0 || alpha_im != 0.0)) {
    h2b_set_error("h2b_bem_new: the single layer operator has no identity term (alpha must be 0)");
    return NULL;
  }
  h2b_bem *b = new h2b_bem();
  b->s = s;
  b->pde = pde;
  b->layer = layer;
  b->row_basis = row_basis;
  b->col_basis = col_basis;
  b->q = q_regular;
  b->q2 = q_singular;
  b->k_re = k_re;
  b->k_im = k_im;
  b->alpha_re = alpha_re;
  b->alpha_im = alpha_im;
  b->kconst = H2B_KERNEL_CONST;
  // Mass matrices of the reference triangle scaled by the Gram determinant
  // (Library/laplacebem3d.c:926-994): ll 1/12 diagonal, 1/24 off-diagonal; cl / lc 1/6.
  for (int i = 0; i < 9; i++) b->mass[i] = 0.0;
  if (row_basis == H2B_BASIS_LINEAR && col_basis == H2B_BASIS_LINEAR) {
    for (int i = 0; i < 3; i++)
      for (int j = 0; j < 3; j++) b->mass[i + 3 * j] = (i == j) ? 1.0 / 12.0 : 1.0 / 24.0;
  } else if (row_basis != col_basis) {
    for (int i = 0; i < 3; i++) b->mass[i] = 1.0 / 6.0;
  }
  if (h2b_quad_build(q_regular, q_singular, row_basis, col_basis, &b->quad) != H2B_OK) {
    delete b;
    return NULL;
  }
  // Packed singular rules for the device, every block padded to an even number of doubles
  // (16-byte alignment).  Case 1 (common vertex): for q_singular = 4 the tensor form of
  // h2b_quad_vert_tensor (rule_n[1] = groups), otherwise x0, x1, y0, y1, w (raw), n_1 doubles
  // each.  Cases 2 and 3 (common edge, identical): the reduced rules of h2b_quad_reduce, a, b, c and
  // the basis-weighted weight rows (i + NR j) for the row / column basis functions i < NR,
  // j < NC (NR, NC = 3 for a linear basis, 1 for a constant one), n_c' doubles each.
  std::vector<double> pack;
  b->rule_n[0] = b->rule_off[0] = 0;
  const int NR = row_basis == H2B_BASIS_LINEAR ? 3 : 1, NC = col_basis == H2B_BASIS_LINEAR ? 3 : 1;
  for (int c = 1; c <= 3; c++) {
    const h2b_rule &r = b->quad.rule[c];
    b->rule_off[c] = (uint32_t) pack.size();
    if (c == 1 && q_singular == 4) {
      // tensor form (h2b_quad_vert_tensor): the kernel's specialised path for q2 = 4
      uint32_t ng = 0;
      double *t = nullptr;
      if (h2b_quad_vert_tensor(q_singular, row_basis, col_basis, &ng, &t) != H2B_OK) {
        h2b_bem_del(b);
        return NULL;
      }
      b->rule_n[c] = ng;
      b->vert_tensor = 1;
      pack.insert(pack.end(), t, t + (size_t) (4 + NR + NC) * q_singular * ng);
      free(t);
    } else if (c == 1) {
      b->rule_n[c] = r.n;
      const double *src[5] = {r.x0, r.x1, r.y0, r.y1, r.w + 9ull * r.n};
      for (int f = 0; f < 5; f++) pack.insert(pack.end(), src[f], src[f] + r.n);
    } else {
      uint32_t n = 0;
      double *abc = nullptr, *w9 = nullptr;
      if (h2b_quad_reduce(&r, c, q_singular, &n, &abc, &w9) != H2B_OK) {
        h2b_bem_del(b);
        return NULL;
      }
      b->rule_n[c] = n;
      pack.insert(pack.end(), abc, abc + 3ull * n);
      for (int j = 0; j < NC; j++)
        for (int i = 0; i < NR; i++)
          pack.insert(pack.end(), w9 + (size_t) (i + 3 * j) * n, w9 + (size_t) (i + 3 * j + 1) * n);
      free(abc);
      free(w9);
    }
    // offsets inside the block are multiples of n; keep n even by padding the whole block
    if (pack.size() & 1) pack.push_back(0.0);
  }
  if (q_singular == 4) {
    // slot 4: the common-vertex rule with the radial sum folded into moments
    // (h2b_quad_vert_merged), used for the Laplace kernels
    uint32_t nm = 0;
    double *t = nullptr;
    if (h2b_quad_vert_merged(q_singular, row_basis, col_basis, &nm, &t) != H2B_OK) {
      h2b_bem_del(b);
      return NULL;
    }
    b->rule_off[4] = (uint32_t) pack.size();
    b->rule_n[4] = nm;
    b->vert_merged = 1;
    pack.insert(pack.end(), t, t + (size_t) (4 + 2 * NR + 4 * NC) * nm);
    free(t);
    if (pack.size() & 1) pack.push_back(0.0);
  }
  // every field must start on a 16-byte boundary: n is a multiple of 2 (2 q2^4 and 6 q2^4)
  b->rule_total = (uint32_t) pack.size();
  cudaStream_t st = b->s->stream;
  if (cudaMallocAsync(&b->d_rule, sizeof(double) * pack.size(), st) != cudaSuccess ||
      cudaMemcpyAsync(b->d_rule, pack.data(), sizeof(double) * pack.size(),
                      cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMallocAsync(&b->d_err, sizeof(int), st) != cudaSuccess ||
      cudaMemsetAsync(b->d_err, 0, sizeof(int), st) != cudaSuccess ||
      cudaEventCreate(&b->ev[0]) != cudaSuccess || cudaEventCreate(&b->ev[1]) != cudaSuccess ||
      cudaEventCreate(&b->ev[2]) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
    h2b_set_error("h2b_bem_new: %s", cudaGetErrorString(cudaGetLastError()));
    h2b_bem_del(b);
    return NULL;
  }
  return b;
}

extern "C" void h2b_bem_del(h2b_bem *b) {
  if (!b) return;
  // the operator must be deleted before its surface (the frees are ordered on its stream)
  if (b->d_rule) cudaFreeAsync(b->d_rule, b->s->stream);
  if (b->d_err) cudaFreeAsync(b->d_err, b->s->stream);
  for (int i = 0; i < 3; i++)
    if (b->ev[i]) cudaEventDestroy(b->ev[i]);
  h2b_quad_free(&b->quad);
  delete b;
}

int h2b_bem_kernel_kind(const h2b_bem *b) {
  if (b->pde == H2B_LAPLACE)
    return b->layer == H2B_SLP ? H2B_KK_LSLP : b->layer == H2B_DLP ? H2B_KK_LDLP : H2B_KK_LADLP;
  return b->layer == H2B_SLP ? H2B_KK_HSLP : b->layer == H2B_DLP ? H2B_KK_HDLP : H2B_KK_HADLP;
}

void h2b_fill_launch(const h2b_bem *b, h2b_near_launch *L) {
  memset(L, 0, sizeof(*L));
  L->kk = h2b_bem_kernel_kind(b);
  L->row_linear = b->row_basis == H2B_BASIS_LINEAR;
  L->col_linear = b->col_basis == H2B_BASIS_LINEAR;
  L->q = b->q;
  L->tri = b->s->d_tri;
  L->qrec = b->s->d_qrec;
  L->kconst = b->kconst;
  L->k_re = b->k_re;
  L->k_imn = -b->k_im;
  L->alpha_re = b->alpha_re;
  L->alpha_im = b->alpha_im;
  for (int i = 0; i < 9; i++) L->mass[i] = b->mass[i];
  L->rule = b->d_rule;
  for (int i = 0; i < 5; i++) {
    L->rule_n[i] = b->rule_n[i];
    L->rule_off[i] = b->rule_off[i];
  }
  L->rule_total = b->rule_total;
  L->vert_tensor = b->vert_tensor;
  L->vert_merged = b->vert_merged;
  L->num_sms = b->s->num_sms;
  L->err = b->d_err;
  L->nvert = UINT32_MAX;
}

uint32_t h2b_bem_rows(const h2b_bem *b) {
  return b->row_basis == H2B_BASIS_LINEAR ? b->s->nv : b->s->nt;
}
uint32_t h2b_bem_cols(const h2b_bem *b) {
  return b->col_basis == H2B_BASIS_LINEAR ? b->s->nv : b->s->nt;
}

// The tiles of one block (rows x cols indices in tiles of `tile`) on the device: the host lists the
// triangles of each side's parts, the tiles themselves are written by a kernel (a dense matrix of
// 8192 indices has 16384 of them, which took 0.4 ms on the host).  Device arrays in *dp, freed by
// h2b_devplan_free.
static int block_plan(const h2b_bem *bem, const uint32_t *ridx, uint32_t rows, const uint32_t *cidx,
                      uint32_t cols, uint32_t ld, int ntrans, uint32_t tile, bool same, cudaStream_t st,
                      h2b_devplan *dp) {
  memset(dp, 0, sizeof(*dp));
  h2b_adjacency *adj = const_cast<h2b_adjacency *>(&bem->s->adj);
  const uint32_t nr = (rows + tile - 1) / tile, nc = (cols + tile - 1) / tile;
  if ((uint64_t) nr * nc > UINT32_MAX / 2) {
    h2b_set_error("h2b_bem_nearfield: %u x %u entries are too many for one call", rows, cols);
    return H2B_ERR_ARG;
  }
  struct Plan : h2b_nearplan {
    Plan() { h2b_nearplan_init(this); }
    ~Plan() { h2b_nearplan_free(this); }
  } plan;
  std::vector<uint32_t> lists(2ull * (nr + nc));
  const int rl = bem->row_basis == H2B_BASIS_LINEAR, cl = bem->col_basis == H2B_BASIS_LINEAR;
  int rc = H2B_OK;
  for (uint32_t i = 0; rc == H2B_OK && i < nr; i++)
    rc = h2b_nearplan_tile_list(&plan, adj, rl, ridx + (size_t) i * tile,
                                std::min(tile, rows - i * tile), &lists[i], &lists[nr + i]);
  for (uint32_t j = 0; rc == H2B_OK && j < nc; j++)
    rc = h2b_nearplan_tile_list(&plan, adj, cl, cidx + (size_t) j * tile,
                                std::min(tile, cols - j * tile), &lists[2 * nr + j],
                                &lists[2 * nr + nc + j]);
  if (rc != H2B_OK) {
    h2b_set_error("h2b_bem_nearfield: out of host memory building the plan");
    return rc;
  }
  dp->ntiles = nr * nc;
  dp->nhalf = same ? nr * (nr + 1) / 2 : 0;
  uint32_t *d_lists = nullptr;
  if (cudaMallocAsync((void **) &dp->tiles, sizeof(h2b_tile) * dp->ntiles, st) != cudaSuccess ||
      (same && cudaMallocAsync((void **) &dp->half, sizeof(uint32_t) * dp->nhalf, st) != cudaSuccess) ||
      cudaMallocAsync((void **) &dp->refs, sizeof(h2b_triref) * std::max(1u, plan.nrefs), st) != cudaSuccess ||
      cudaMemcpyAsync(dp->refs, plan.refs, sizeof(h2b_triref) * plan.nrefs, cudaMemcpyHostToDevice,
                      st) != cudaSuccess ||
      cudaMallocAsync((void **) &d_lists, sizeof(uint32_t) * lists.size(), st) != cudaSuccess ||
      cudaMemcpyAsync(d_lists, lists.data(), sizeof(uint32_t) * lists.size(),
                      cudaMemcpyHostToDevice, st) != cudaSuccess) {
    h2b_set_error("h2b_bem_nearfield: %s", cudaGetErrorString(cudaGetLastError()));
    rc = H2B_ERR_CUDA;
  }
  if (rc == H2B_OK)
    rc = h2b_near_grid_tiles(d_lists, nr, nc, rows, cols, tile, ld, ntrans, dp->tiles, dp->half, st);
  if (d_lists) cudaFreeAsync(d_lists, st);
  return rc;
}

int h2b_classify_device(const h2b_surface *s, const void *refs, const h2b_tile *tiles,
                        uint32_t ntiles, cudaStream_t st, h2b_sing **d_sing, uint32_t cnt[4]) {
  *d_sing = nullptr;
  for (int c = 0; c < 4; c++) cnt[c] = 0;
  uint32_t *d_cur = nullptr;
  H2B_CUDA_TRY(cudaMallocAsync(&d_cur, sizeof(uint32_t) * 8, st));
  int rc = H2B_OK;
  // d_cur[0..3]: pairs per case of the count pass, [4..7]: the write pass's cursors
  uint32_t host[4] = {0, 0, 0, 0};
  if (cudaMemsetAsync(d_cur, 0, sizeof(uint32_t) * 8, st) != cudaSuccess) rc = H2B_ERR_CUDA;
  if (rc == H2B_OK)
    rc = h2b_near_classify(s->d_tri, refs, tiles, ntiles, s->d_nb_off, s->d_nb_len, s->d_nb, d_cur,
                           nullptr, nullptr, st);
  if (rc == H2B_OK &&
      (cudaMemcpyAsync(host, d_cur, sizeof(uint32_t) * 4, cudaMemcpyDeviceToHost, st) !=
           cudaSuccess ||
       cudaStreamSynchronize(st) != cudaSuccess))
    rc = H2B_ERR_CUDA;
  const uint64_t nsing = (uint64_t) host[1] + host[2] + host[3];
  if (rc == H2B_OK && nsing > UINT32_MAX) {
    h2b_set_error("singular-pair classification: %llu pairs exceed the 32-bit pair list",
                  (unsigned long long) nsing);
    cudaFreeAsync(d_cur, st);
    return H2B_ERR_ARG;
  }
  if (rc == H2B_OK && nsing &&
      cudaMallocAsync((void **) d_sing, sizeof(h2b_sing) * nsing, st) != cudaSuccess)
    rc = H2B_ERR_CUDA;
  if (rc == H2B_OK && nsing)
    rc = h2b_near_classify(s->d_tri, refs, tiles, ntiles, s->d_nb_off, s->d_nb_len, s->d_nb, d_cur + 4,
                           d_cur, *d_sing, st);
  if (rc == H2B_ERR_CUDA)
    h2b_set_error("singular-pair classification: %s", cudaGetErrorString(cudaGetLastError()));
  cudaFreeAsync(d_cur, st);
  if (rc != H2B_OK && *d_sing) {
    cudaFreeAsync(*d_sing, st);
    *d_sing = nullptr;
  }
  if (rc == H2B_OK)
    for (int c = 1; c <= 3; c++) cnt[c] = host[c];
  return rc;
}

void h2b_devplan_free(h2b_devplan *dp, cudaStream_t st) {
  if (dp->tiles) cudaFreeAsync(dp->tiles, st);
  if (dp->half) cudaFreeAsync(dp->half, st);
  if (dp->refs) cudaFreeAsync(dp->refs, st);
  if (dp->sing) cudaFreeAsync(dp->sing, st);
  memset(dp, 0, sizeof(*dp));
}

int h2b_check_err_flag(const h2b_bem *b, cudaStream_t st) {
  int flag = 0;
  H2B_CUDA_TRY(cudaMemcpyAsync(&flag, b->d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
  H2B_CUDA_TRY(cudaStreamSynchronize(st));
  if (flag) {
    h2b_set_error("quadrature kernel: staging of the singular rules timed out");
    cudaMemsetAsync(b->d_err, 0, sizeof(int), st);
    return H2B_ERR_TIMEOUT;
  }
  return H2B_OK;
}

// ------------------------------------------------------------------------------------------
// Nearfield blocks
// ------------------------------------------------------------------------------------------

// Tile size of a block: the one with the least estimated time, rounds of the SMs (1.5 resident tiles
// each, measured between one and two) times the lanes a tile's triangle pairs take.  A tile side of
// s vertices touches about 2 s + 4.3 sqrt(s) triangles (the inner ones and those along the border,
// counted on refined spheres), rows in groups of 32 lanes, so smaller tiles evaluate border pairs more
// often but spread a small block over the SMs; with constant bases tiles share no pairs.  Linear
// columns with q = 2 spread a tile over a cluster of up to eight CTAs as well (near_ring_kernel).  The
// estimate fills two CTAs per SM three times over, as the launch does (RING_FILL) for kernels of up to
// three planes; the launch of the complex double layer with mates counts one CTA per SM.  FIXED is the fixed cost of a tile in pairs (clearing, staging and writing
// it).  60 x 57 linear block: four tiles of 32 take 46 us, 8 x 8 tiles 16 us, with clusters 10.
// 578 x 578 complex double layer, us: a CTA per tile of 16 613, of 32 533 to 642; a
// cluster per tile of 64 421.
static uint32_t block_tile(const h2b_bem *b, uint32_t rows, uint32_t cols, bool same) {
  constexpr double FIXED = 400.0;
  const bool rl = b->row_basis == H2B_BASIS_LINEAR, cl = b->col_basis == H2B_BASIS_LINEAR;
  uint32_t best = H2B_TILE_MAX;
  double least = 0.0;
  for (uint32_t t = H2B_TILE_MAX; t >= 8; t /= 2) {
    auto tri = [&](uint32_t n, bool lin) {
      const double s = n < t ? n : t;
      return lin ? 2.0 * s + 4.3 * sqrt(s) : s;
    };
    double r = tri(rows, rl);
    if (cl) r = 32.0 * ceil(r / 32.0);
    double n = ceil((double) rows / t) * ceil((double) cols / t);
    if (same) n = 0.5 * (n + ceil((double) rows / t));
    double work = r * tri(cols, cl);
    if (cl && b->q == 2)
      for (int share = 1; share < 8 && 2.0 * n <= 6.0 * b->s->num_sms; share *= 2) n *= 2, work /= 2;
    const double rounds = n / (1.5 * b->s->num_sms);
    const double cost = (rounds > 1.0 ? rounds : 1.0) * (work + FIXED);
    if (t == H2B_TILE_MAX || cost < 0.9 * least) {
      best = t;
      least = cost;
    }
  }
  return best;
}

extern "C" int h2b_bem_nearfield(const h2b_bem *bem, const uint32_t *ridx, uint32_t rows,
                                 const uint32_t *cidx, uint32_t cols, int ntrans, double *N,
                                 uint64_t ld) {
  if (!bem || !N) {
    h2b_set_error("h2b_bem_nearfield: NULL operator or output");
    return H2B_ERR_ARG;
  }
  if (rows == 0 || cols == 0) return H2B_OK;
  const uint32_t out_rows = ntrans ? cols : rows, out_cols = ntrans ? rows : cols;
  if (ld < out_rows) {
    h2b_set_error("h2b_bem_nearfield: ld %llu < %u rows of the output",
                  (unsigned long long) ld, out_rows);
    return H2B_ERR_ARG;
  }
  int rc = h2b_ensure_device();
  if (rc != H2B_OK) return rc;
  const h2b_surface *s = bem->s;
  const uint32_t nr_all = h2b_bem_rows(bem), nc_all = h2b_bem_cols(bem);
  std::vector<uint32_t> ri, ci;
  if (!ridx) {
    ri.resize(rows);
    for (uint32_t i = 0; i < rows; i++) ri[i] = i;
    ridx = ri.data();
  }
  if (!cidx) {
    ci.resize(cols);
    for (uint32_t i = 0; i < cols; i++) ci[i] = i;
    cidx = ci.data();
  }
  // validate indices and reject duplicates (H2Lib index sets are permutations)
  {
    std::vector<uint8_t> seen(nr_all > nc_all ? nr_all : nc_all, 0);
    for (uint32_t i = 0; i < rows; i++) {
      if (ridx[i] >= nr_all || seen[ridx[i]]) {
        h2b_set_error("h2b_bem_nearfield: row index %u invalid or repeated", ridx[i]);
        return H2B_ERR_ARG;
      }
      seen[ridx[i]] = 1;
    }
    std::fill(seen.begin(), seen.end(), 0);
    for (uint32_t i = 0; i < cols; i++) {
      if (cidx[i] >= nc_all || seen[cidx[i]]) {
        h2b_set_error("h2b_bem_nearfield: column index %u invalid or repeated", cidx[i]);
        return H2B_ERR_ARG;
      }
      seen[cidx[i]] = 1;
    }
  }
  const int cplx = bem->pde == H2B_HELMHOLTZ;
  const size_t es = cplx ? 16 : 8;
  cudaStream_t st = s->stream;
  const bool dev_out = h2b_is_device_ptr(N);
  const uint64_t ld_dev = dev_out ? ld : out_rows;

  const bool same = bem->row_basis == bem->col_basis && rows == cols &&
                    !memcmp(ridx, cidx, sizeof(uint32_t) * rows);
  if (same) cidx = ridx;  // one set of triangle lists
  const uint32_t tile = block_tile(bem, rows, cols, same);

  h2b_devplan dp;
  rc = block_plan(bem, ridx, rows, cidx, cols, (uint32_t) ld_dev, ntrans, tile, same, st, &dp);
  if (rc != H2B_OK) {
    h2b_devplan_free(&dp, st);
    return rc;
  }
  {
    uint32_t cnt[4];
    rc = h2b_classify_device(s, dp.refs, dp.tiles, dp.ntiles, st, &dp.sing, cnt);
    if (rc != H2B_OK) {
      h2b_devplan_free(&dp, st);
      return rc;
    }
    dp.nsing = cnt[1] + cnt[2] + cnt[3];
    dp.nvert = cnt[1];
  }

  double *out = N;
  if (!dev_out) {
    if (cudaMallocAsync((void **) &out, es * ld_dev * out_cols, st) != cudaSuccess) {
      h2b_devplan_free(&dp, st);
      h2b_set_error("h2b_bem_nearfield: device allocation of %llu bytes failed",
                    (unsigned long long) (es * ld_dev * out_cols));
      return H2B_ERR_NOMEM;
    }
  }
  h2b_near_launch L;
  h2b_fill_launch(bem, &L);
  L.refs = dp.refs;
  L.tiles = dp.tiles;
  L.ntiles = dp.ntiles;
  L.half = dp.half;
  L.nhalf = dp.nhalf;
  L.sing = dp.sing;
  L.nsing = dp.nsing;
  L.nvert = dp.nvert;
  L.out0 = out;
  // the operator's own events time the two kernels (nearfield diagnostics, h2b_bem_timings)
  h2b_bem *mb = const_cast<h2b_bem *>(bem);
  L.ev_between = mb->ev[1];
  if (cudaEventRecord(mb->ev[0], st) != cudaSuccess) rc = H2B_ERR_CUDA;
  if (rc == H2B_OK) rc = h2b_near_launch_kernels(&L, st);
  if (rc == H2B_OK && cudaEventRecord(mb->ev[2], st) != cudaSuccess) rc = H2B_ERR_CUDA;
  if (rc == H2B_OK && !dev_out) {
    if (cudaMemcpy2DAsync(N, ld * es, out, ld_dev * es, out_rows * es, out_cols,
                          cudaMemcpyDeviceToHost, st) != cudaSuccess) {
      h2b_set_error("h2b_bem_nearfield: copy back failed: %s",
                    cudaGetErrorString(cudaGetLastError()));
      rc = H2B_ERR_CUDA;
    }
  }
  if (!dev_out) cudaFreeAsync(out, st);
  h2b_devplan_free(&dp, st);
  if (rc == H2B_OK) rc = h2b_check_err_flag(bem, st);
  if (cudaStreamSynchronize(st) != cudaSuccess && rc == H2B_OK) {
    h2b_set_error("h2b_bem_nearfield: %s", cudaGetErrorString(cudaGetLastError()));
    rc = H2B_ERR_CUDA;
  }
  if (rc == H2B_OK) {
    float a = 0.0f, b = 0.0f;
    // ev[1] is recorded only when the plan has distant tiles; otherwise both phases read 0
    if (cudaEventElapsedTime(&a, mb->ev[0], mb->ev[1]) != cudaSuccess ||
        cudaEventElapsedTime(&b, mb->ev[1], mb->ev[2]) != cudaSuccess) {
      cudaGetLastError();
      a = b = 0.0f;
    }
    mb->near_ms[0] = a;
    mb->near_ms[1] = b;
  }
  return rc;
}

extern "C" int h2b_bem_timings(const h2b_bem *bem, double ms[2]) {
  if (!bem || !ms) return H2B_ERR_ARG;
  ms[0] = bem->near_ms[0];
  ms[1] = bem->near_ms[1];
  return H2B_OK;
}

extern "C" int h2b_bem_assemble_amatrix(const h2b_bem *bem, double *G, uint64_t ld) {
  if (!bem) {
    h2b_set_error("h2b_bem_assemble_amatrix: NULL operator");
    return H2B_ERR_ARG;
  }
  // Like assemble_bem3d_amatrix (Library/bem3d.c:9988) the matrix is square: the column count is
  // taken from the row basis.
  const uint32_t n = h2b_bem_rows(bem);
  if (h2b_bem_cols(bem) != n) {
    h2b_set_error("h2b_bem_assemble_amatrix: row and column index sets differ in size");
    return H2B_ERR_ARG;
  }
  return h2b_bem_nearfield(bem, NULL, n, NULL, n, 0, G, ld);
}
