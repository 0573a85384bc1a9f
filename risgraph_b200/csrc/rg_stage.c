/* Host side of a staged update batch: one pass over the caller's edges that
 * checks them and writes the 32-bit records the device takes (vertex ids are
 * below 2^31, weights fit their codes) into pinned memory.  The caller's
 * records are 24 or 16 bytes of cold memory, so a pass costs what reading them
 * does; separate passes for the check, the weight scan and a plain copy took
 * 0.8 ms for 100,000 edges, this one 0.1. */
#include "rg_stage.h"

/* threads: the steps of a batch from RG_STAGE_PARALLEL edges on are cut over eight
 * threads, the last and smaller one too (262,144 weighted edges: 810 us on one
 * thread, 117 on eight, on a 16-core host). */

/* The top bit of the result is set when an id is not below V (ids above 2^63
 * show in the OR, others in the sign of V - 1 - id). */
#define BAD_IDS(s, d) ((s) | (d) | (last - (s)) | (last - (d)))

int rg_stage_edges(const rg_edge *e, uint64_t n, uint64_t V, int weighted, uint64_t raw_max, uint64_t limit, int threads,
                   uint32_t *out) {
  const uint64_t last = V - 1;
  uint64_t bad = 0, heavy = 0, over = 0;
  const int64_t m = (int64_t)n;
  if (weighted) {
#pragma omp parallel for reduction(| : bad, heavy, over) schedule(static) if (threads) num_threads(8)
    for (int64_t i = 0; i < m; i++) {
      const uint64_t s = e[i].src, d = e[i].dst, w = e[i].data;
      bad |= BAD_IDS(s, d);
      heavy |= w > raw_max;
      over |= w >= limit;
      out[3 * i] = (uint32_t)s;
      out[3 * i + 1] = (uint32_t)d;
      out[3 * i + 2] = (uint32_t)w;
    }
  } else {
#pragma omp parallel for reduction(| : bad) schedule(static) if (threads) num_threads(8)
    for (int64_t i = 0; i < m; i++) {
      const uint64_t s = e[i].src, d = e[i].dst;
      bad |= BAD_IDS(s, d);
      out[2 * i] = (uint32_t)s;
      out[2 * i + 1] = (uint32_t)d;
    }
  }
  return ((bad >> 63) || over ? RG_STAGE_BAD : 0) | (heavy ? RG_STAGE_HEAVY : 0);
}

int rg_stage_pairs(const uint64_t *p, uint64_t n, uint64_t V, int threads, uint32_t *out) {
  const uint64_t last = V - 1;
  uint64_t bad = 0;
  const int64_t m = (int64_t)n;
#pragma omp parallel for reduction(| : bad) schedule(static) if (threads) num_threads(8)
  for (int64_t i = 0; i < m; i++) {
    const uint64_t s = p[2 * i], d = p[2 * i + 1];
    bad |= BAD_IDS(s, d);
    out[2 * i] = (uint32_t)s;
    out[2 * i + 1] = (uint32_t)d;
  }
  return bad >> 63 ? RG_STAGE_BAD : 0;
}
