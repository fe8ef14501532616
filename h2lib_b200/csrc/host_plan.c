/* Host-side nearfield plans: cut the requested blocks into output tiles of at most 64 x 64
 * entries and list the triangles each tile touches.  The device kernels consume the flat arrays; the
 * singular (vertex-sharing) triangle pairs are found on the device (h2b_near_classify).
 *
 * Semantics follow the reference's nearfield callbacks:
 *   constant basis  assemble_cc_near_bem3d   Library/bem3d.c:1151 — one triangle pair per entry;
 *   linear basis    assemble_ll_near_bem3d   Library/bem3d.c:3038 — entry (i, j) sums every pair
 *                   (t, s) with vertex i in t and vertex j in s, using the weight of the local
 *                   basis functions of i in t and j in s; cl / lc mix the two.
 */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include "h2b200_plan.h"

#define GROW(arr, n, cap, extra, type)                                                   \
  do {                                                                                 \
    if ((n) + (extra) > (cap)) {                                                       \
      size_t nc_ = ((size_t) (n) + (extra)) * 2 + 64;                                  \
      type *p_ = (type *) realloc((arr), sizeof(type) * nc_);                          \
      if (!p_) return H2B_ERR_NOMEM;                                                   \
      (arr) = p_;                                                                      \
      (cap) = nc_;                                                                     \
    }                                                                                  \
  } while (0)

int
h2b_adjacency_build(uint32_t vertices, uint32_t triangles, const uint32_t *t, h2b_adjacency *adj)
{
  uint32_t i, k;
  memset(adj, 0, sizeof(*adj));
  adj->nv = vertices;
  adj->nt = triangles;
  adj->off = (uint32_t *) calloc((size_t) vertices + 1, sizeof(uint32_t));
  adj->tri = (uint32_t *) malloc(sizeof(uint32_t) * 3 * (size_t) (triangles ? triangles : 1));
  adj->vstamp = (uint32_t *) calloc(vertices ? vertices : 1, sizeof(uint32_t));
  adj->vloc = (int32_t *) calloc(vertices ? vertices : 1, sizeof(int32_t));
  adj->tstamp = (uint32_t *) calloc(triangles ? triangles : 1, sizeof(uint32_t));
  if (!adj->off || !adj->tri || !adj->vstamp || !adj->vloc || !adj->tstamp) {
    h2b_adjacency_free(adj);
    return H2B_ERR_NOMEM;
  }
  for (i = 0; i < triangles; i++)
    for (k = 0; k < 3; k++)
      adj->off[t[3 * (size_t) i + k] + 1]++;
  for (i = 0; i < vertices; i++)
    adj->off[i + 1] += adj->off[i];
  {
    uint32_t *fill = (uint32_t *) malloc(sizeof(uint32_t) * (vertices ? vertices : 1));
    if (!fill) {
      h2b_adjacency_free(adj);
      return H2B_ERR_NOMEM;
    }
    memcpy(fill, adj->off, sizeof(uint32_t) * vertices);
    for (i = 0; i < triangles; i++)
      for (k = 0; k < 3; k++) {
        uint32_t v = t[3 * (size_t) i + k];
        adj->tri[fill[v]++] = i;
      }
    free(fill);
  }
  adj->t = t;
  adj->gen = 0;
  return H2B_OK;
}

void
h2b_adjacency_free(h2b_adjacency *adj)
{
  free(adj->off); free(adj->tri); free(adj->vstamp); free(adj->vloc); free(adj->tstamp);
  memset(adj, 0, sizeof(*adj));
}

void
h2b_nearplan_init(h2b_nearplan *p)
{
  memset(p, 0, sizeof(*p));
}

void
h2b_nearplan_free(h2b_nearplan *p)
{
  free(p->tiles); free(p->refs);
  free((void *) p->lkey); free(p->lkn); free(p->loff); free(p->llen);
  free(p->order);
  memset(p, 0, sizeof(*p));
}

static size_t
list_slot(const h2b_nearplan *p, const uint32_t *idx, uint32_t kn)
{
  size_t h = ((size_t) (uintptr_t) idx >> 2) * 0x9E3779B97F4A7C15ull ^ (size_t) kn * 0xC2B2AE3D27D4EB4Full;
  size_t m = p->lcap - 1, i = (h >> 17) & m;
  while (p->lkey[i] && !(p->lkey[i] == idx && p->lkn[i] == kn))
    i = (i + 1) & m;
  return i;
}

/* Grow the list table to keep it at most half full. */
static int
list_reserve(h2b_nearplan *p)
{
  size_t i, oc = p->lcap;
  const uint32_t **ok = p->lkey;
  uint32_t *okn = p->lkn, *ooff = p->loff, *olen = p->llen;
  if (2 * (p->lcount + 1) <= p->lcap)
    return H2B_OK;
  p->lcap = oc ? 2 * oc : 1024;
  p->lkey = (const uint32_t **) calloc(p->lcap, sizeof(*p->lkey));
  p->lkn = (uint32_t *) calloc(p->lcap, sizeof(uint32_t));
  p->loff = (uint32_t *) calloc(p->lcap, sizeof(uint32_t));
  p->llen = (uint32_t *) calloc(p->lcap, sizeof(uint32_t));
  if (!p->lkey || !p->lkn || !p->loff || !p->llen)
    return H2B_ERR_NOMEM;
  for (i = 0; i < oc; i++)
    if (ok[i]) {
      size_t j = list_slot(p, ok[i], okn[i]);
      p->lkey[j] = ok[i];
      p->lkn[j] = okn[i];
      p->loff[j] = ooff[i];
      p->llen[j] = olen[i];
    }
  free((void *) ok); free(okn); free(ooff); free(olen);
  return H2B_OK;
}

static uint32_t
next_gen(h2b_adjacency *adj)
{
  if (++adj->gen == 0) {   /* wrapped: reset stamps */
    memset(adj->vstamp, 0, sizeof(uint32_t) * adj->nv);
    memset(adj->tstamp, 0, sizeof(uint32_t) * adj->nt);
    adj->gen = 1;
  }
  return adj->gen;
}

/* Orders the triangles of a linear list by id and assigns their vertices to three slots: the
 * distant-pair kernel walks along the list and keeps the sums of a vertex in registers while
 * consecutive triangles share it.  Refined and generated meshes number neighbouring triangles
 * consecutively, so the walk leaves 0.8 vertices per triangle on a refined sphere (2.3 of a
 * triangle's vertices lie in the cluster); a greedy strip over the list leaves 0.75. */
static int
order_list(h2b_nearplan *p, const h2b_adjacency *adj, uint32_t off, uint32_t n)
{
  h2b_triref *r = p->refs + off, *tmp;
  uint64_t *src, *dst;
  uint32_t i, held[3] = {UINT32_MAX, UINT32_MAX, UINT32_MAX};
  const size_t need = 2 * (size_t) n + (sizeof(h2b_triref) * (size_t) n + 7) / 8;
  if (need > p->corder) {
    uint64_t *o = (uint64_t *) realloc(p->order, sizeof(uint64_t) * 2 * need);
    if (!o)
      return H2B_ERR_NOMEM;
    p->order = o;
    p->corder = 2 * need;
  }
  /* (id, position) sorted by merging ascending runs: the list comes in one run per vertex */
  src = p->order;
  dst = src + n;
  for (i = 0; i < n; i++)
    src[i] = (uint64_t) r[i].t << 32 | i;
  for (;;) {
    uint32_t o = 0, runs = 0;
    uint64_t *swap;
    while (o < n) {
      uint32_t x = o, m = o + 1, y, e, w = o;
      while (m < n && src[m] > src[m - 1])
        m++;
      for (e = y = m; e < n && (e == m || src[e] > src[e - 1]); e++)
        ;
      while (x < m && y < e)
        dst[w++] = src[x] < src[y] ? src[x++] : src[y++];
      while (x < m)
        dst[w++] = src[x++];
      while (y < e)
        dst[w++] = src[y++];
      o = e;
      runs++;
    }
    swap = src;
    src = dst;
    dst = swap;
    if (runs <= 1)
      break;
  }
  tmp = (h2b_triref *) (p->order + 2 * (size_t) n);
  memcpy(tmp, r, sizeof(*r) * n);
  for (i = 0; i < n; i++) {
    const uint32_t *v;
    int at[3] = {-1, -1, -1}, j, s;
    uint32_t placed = 0;
    r[i] = tmp[(uint32_t) src[i]];
    v = adj->t + 3 * (size_t) r[i].t;
    for (j = 0; j < 3; j++)
      for (s = 0; s < 3; s++)
        if (at[s] < 0 && v[j] == held[s]) {
          at[s] = j;
          placed |= 1u << j;
          break;
        }
    for (j = 0; j < 3; j++)
      if (!(placed >> j & 1u)) {
        for (s = 0; at[s] >= 0; s++)
          ;
        at[s] = j;
      }
    for (s = 0; s < 3; s++)
      held[s] = v[at[s]];
    r[i].slots = (int16_t) (at[0] | at[1] << 2 | at[2] << 4);
  }
  return H2B_OK;
}

/* Append the triangle list of an index range; returns its offset in p->refs. */
static int
add_reflist(h2b_nearplan *p, h2b_adjacency *adj, int linear, const uint32_t *idx, uint32_t n,
            uint32_t *off, uint32_t *len)
{
  uint32_t i, k;
  *off = p->nrefs;
  if (!linear) {
    GROW(p->refs, p->nrefs, p->crefs, n, h2b_triref);
    for (i = 0; i < n; i++) {
      h2b_triref *r = &p->refs[p->nrefs++];
      r->t = idx[i];
      r->l[0] = r->l[1] = r->l[2] = (int16_t) i;
      r->slots = 0;
    }
  }
  else {
    uint32_t gv = next_gen(adj), gt;
    for (i = 0; i < n; i++) {
      adj->vstamp[idx[i]] = gv;
      adj->vloc[idx[i]] = (int32_t) i;
    }
    gt = next_gen(adj);
    /* vertex stamps of the first generation stay valid: compare against gv below */
    for (i = 0; i < n; i++) {
      uint32_t v = idx[i], a;
      for (a = adj->off[v]; a < adj->off[v + 1]; a++) {
        uint32_t tt = adj->tri[a];
        h2b_triref *r;
        if (adj->tstamp[tt] == gt)
          continue;
        adj->tstamp[tt] = gt;
        GROW(p->refs, p->nrefs, p->crefs, 1, h2b_triref);
        r = &p->refs[p->nrefs++];
        r->t = tt;
        for (k = 0; k < 3; k++) {
          uint32_t w = adj->t[3 * (size_t) tt + k];
          r->l[k] = (adj->vstamp[w] == gv) ? (int16_t) adj->vloc[w] : (int16_t) -1;
        }
        r->slots = 0;
      }
    }
  }
  *len = p->nrefs - *off;
  return H2B_OK;
}

int
h2b_nearplan_add_reflist(h2b_nearplan *p, h2b_adjacency *adj, int linear, const uint32_t *idx,
                         uint32_t n, uint32_t *off, uint32_t *len)
{
  return add_reflist(p, adj, linear, idx, n, off, len);
}

/* add_reflist, reusing the list of an index range seen before. */
static int
cached_reflist(h2b_nearplan *p, h2b_adjacency *adj, int linear, const uint32_t *idx, uint32_t n,
               uint32_t *off, uint32_t *len)
{
  const uint32_t kn = (n << 1) | (linear ? 1u : 0u);
  size_t i;
  int rc;
  if ((rc = list_reserve(p)) != H2B_OK)
    return rc;
  i = list_slot(p, idx, kn);
  if (p->lkey[i]) {
    *off = p->loff[i];
    *len = p->llen[i];
    return H2B_OK;
  }
  if ((rc = add_reflist(p, adj, linear, idx, n, off, len)) != H2B_OK)
    return rc;
  if (linear && (rc = order_list(p, adj, *off, *len)) != H2B_OK)
    return rc;
  p->lkey[i] = idx;
  p->lkn[i] = kn;
  p->loff[i] = *off;
  p->llen[i] = *len;
  p->lcount++;
  return H2B_OK;
}

int
h2b_nearplan_tile_list(h2b_nearplan *p, h2b_adjacency *adj, int linear, const uint32_t *idx,
                       uint32_t n, uint32_t *off, uint32_t *len)
{
  return cached_reflist(p, adj, linear, idx, n, off, len);
}

static int
add_tile(h2b_nearplan *p, h2b_adjacency *adj, int row_linear, int col_linear,
         const uint32_t *ridx, uint32_t rows, const uint32_t *cidx, uint32_t cols,
         uint64_t out_off, uint32_t ld, int ntrans)
{
  h2b_tile *tl;
  uint32_t tr_off, tr_len, sc_off, sc_len;
  int rc;

  if ((rc = cached_reflist(p, adj, row_linear, ridx, rows, &tr_off, &tr_len)) != H2B_OK)
    return rc;
  if ((rc = cached_reflist(p, adj, col_linear, cidx, cols, &sc_off, &sc_len)) != H2B_OK)
    return rc;

  GROW(p->tiles, p->ntiles, p->ctiles, 1, h2b_tile);
  tl = &p->tiles[p->ntiles];
  tl->tr_off = tr_off;
  tl->tr_len = tr_len;
  tl->sc_off = sc_off;
  tl->sc_len = sc_len;
  tl->out_off = out_off;
  tl->ld = ld;
  tl->rows = (uint16_t) rows;
  tl->cols = (uint16_t) cols;
  tl->flags = ntrans ? 1u : 0u;
  tl->mate = 0;
  p->ntiles++;
  return H2B_OK;
}

int
h2b_nearplan_add_block(h2b_nearplan *p, h2b_adjacency *adj, int row_basis, int col_basis,
                       const uint32_t *ridx, uint32_t rows, const uint32_t *cidx, uint32_t cols,
                       uint64_t out_off, uint32_t ld, int ntrans, uint32_t tile)
{
  int rl = (row_basis == H2B_BASIS_LINEAR), cl = (col_basis == H2B_BASIS_LINEAR);
  uint32_t r0, c0;
  if (tile == 0 || tile > H2B_TILE_MAX)
    tile = H2B_TILE_MAX;
  for (c0 = 0; c0 < cols; c0 += tile) {
    uint32_t nc = cols - c0 < tile ? cols - c0 : tile;
    for (r0 = 0; r0 < rows; r0 += tile) {
      uint32_t nr = rows - r0 < tile ? rows - r0 : tile;
      uint64_t off = ntrans ? out_off + c0 + (uint64_t) r0 * ld : out_off + r0 + (uint64_t) c0 * ld;
      int rc = add_tile(p, adj, rl, cl, ridx + r0, nr, cidx + c0, nc, off, ld, ntrans);
      if (rc != H2B_OK)
        return rc;
    }
  }
  return H2B_OK;
}

void
h2b_nearplan_mate(h2b_nearplan *p, uint32_t t0, uint32_t t1, uint32_t nr, uint32_t nc)
{
  uint32_t i, j;
  for (j = 0; j < nc; j++)
    for (i = 0; i < nr; i++) {
      const uint32_t a = t0 + i + j * nr, b = t1 + j + i * nc;
      if (a == b)
        continue;
      p->tiles[a].mate = b + 1;
      p->tiles[b].mate = a + 1;
    }
}

uint32_t
h2b_nearplan_halves(const h2b_nearplan *p, uint32_t *list)
{
  uint32_t cnt[8] = {0}, start[8], i, b, n = 0;
  uint64_t most = 1;
#define WORK(T) ((uint64_t) (T).tr_len * (T).sc_len)
#define SKIP(I) (p->tiles[I].mate && p->tiles[I].mate - 1 < (I))
  for (i = 0; i < p->ntiles; i++)
    if (WORK(p->tiles[i]) > most)
      most = WORK(p->tiles[i]);
  for (i = 0; i < p->ntiles; i++)
    if (!SKIP(i))
      cnt[7 - (WORK(p->tiles[i]) * 7 + most - 1) / most]++;
  for (b = 0; b < 8; b++) {
    start[b] = n;
    n += cnt[b];
  }
  for (i = 0; i < p->ntiles; i++)
    if (!SKIP(i))
      list[start[7 - (WORK(p->tiles[i]) * 7 + most - 1) / most]++] = i;
#undef SKIP
#undef WORK
  return n;
}
