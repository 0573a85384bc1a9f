/* Host staging of update batches (rg_stage.c). */
#ifndef RG_STAGE_H
#define RG_STAGE_H
#include <stdint.h>

#include "risgraph_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* What a pass found: an id >= V or a weight >= limit; a weight above raw_max. */
enum { RG_STAGE_BAD = 1, RG_STAGE_HEAVY = 2 };

/* Batches of at least this many edges are packed by several threads. */
#define RG_STAGE_PARALLEL (1u << 18)

/* n edges to {src, dst, weight} (weighted) or {src, dst} records of 32-bit
 * words at out.  Records of a batch that is BAD or HEAVY are not to be used. */
__attribute__((visibility("hidden"))) int rg_stage_edges(const rg_edge *e, uint64_t n, uint64_t V, int weighted,
                                                         uint64_t raw_max, uint64_t limit, int threads,
                                                         uint32_t *out);
/* n (src, dst) pairs to {src, dst} records. */
__attribute__((visibility("hidden"))) int rg_stage_pairs(const uint64_t *p, uint64_t n, uint64_t V, int threads,
                                                         uint32_t *out);

#ifdef __cplusplus
}
#endif
#endif
