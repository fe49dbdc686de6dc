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

#ifdef __cplusplus
}
#endif

#endif
