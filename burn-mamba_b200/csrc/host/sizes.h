/* Least workspace of the SSD calls, asked by the host path (native.cpp) when memory does not hold what the bm_*_workspace_bytes
 * queries say: not part of the C ABI.  Every bm_ssd* call runs with any size from this one on. */
#ifndef BM_B200_SIZES_HOST_H
#define BM_B200_SIZES_HOST_H

#include <stddef.h>

#include "../../../include/bm_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

size_t bmx_ssd2_fwd_least_bytes(const bm_ssd2_fwd_args* a);
size_t bmx_ssd3_fwd_least_bytes(const bm_ssd3_fwd_args* a);
size_t bmx_ssd2_bwd_least_bytes(const bm_ssd2_bwd_args* a);
size_t bmx_ssd3_bwd_least_bytes(const bm_ssd3_bwd_args* a);

#ifdef __cplusplus
}
#endif
#endif
