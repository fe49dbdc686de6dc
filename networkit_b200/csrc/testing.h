/* Entry points of libnkgpu for its own tests; not part of the C ABI. */
#ifndef NKG_TESTING_H
#define NKG_TESTING_H

#include <stdint.h>

#include "nkgpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* The calling thread's device allocation number `after` from now (0: the next
 * one) fails once with NKG_ERR_OOM, as if memory had run out; negative: none.
 * Returns how many were still to come before the failure set earlier
 * (negative: it has happened, or none was set). */
NKG_API int64_t nkg_test_fail_alloc(int64_t after);

/* For the one-launch runs of this graph: polls of the grid barrier before it
 * gives up (0: at once), and the launch's CTAs (0: as many as the graph needs).
 * Before the handle's first run. */
NKG_API void nkg_test_small_run(nkg_graph *g, uint32_t polls, uint32_t ctas);

/* Graphs of more than `nodes` nodes go to the kernel that nkg_batch_tuning
 * applies to (0: every graph). Before the handle's first run. */
NKG_API void nkg_test_batch_shared(nkg_batch *b, uint32_t nodes);

#ifdef __cplusplus
}
#endif

#endif
