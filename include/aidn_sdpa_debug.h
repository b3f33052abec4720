/*
 * aidn_sdpa_debug.h — test and development hook of libaidotnet_sdpa_sm100.  Not part of the drop-in surface: nothing in
 * the reference binds it and a production caller never needs it.  No counterpart in the reference.
 */
#ifndef AIDN_SDPA_DEBUG_H_
#define AIDN_SDPA_DEBUG_H_

#include "aidn_sdpa.h"

#ifdef __cplusplus
extern "C" {
#endif

/* mode 0: off.
 * mode 3: the producers of the tcgen05 kernels of this handle (prefill, backward, projection GEMM, in 16 bits and in fp32)
 *         withhold their loads and every bounded device-side wait gives up after 20 ms instead of 2 s, so that a test can watch
 *         aidn_sdpa_poll report AIDN_ETIMEOUT and the next launch succeed — without any fault on the device.  `buf`
 *         is ignored.
 *         With a null handle: the calling thread's next aidn_qkv_rope_cache does so, and aidn_qkv_rope_poll reports it
 *         (mode 0 takes that back).
 * modes 1, 2 and 4 exist only in development builds of the library (compiled with -DAIDN_PREFILL_TRACE=1): value tap,
 *         per-work-item timeline and per-step clock stamps of the prefill kernel, written to `buf`.  The shipped build
 *         ignores them. */
AIDN_API int aidn_sdpa_debug_set(aidn_sdpa_t h, float* buf, int mode);

#ifdef __cplusplus
}
#endif
#endif /* AIDN_SDPA_DEBUG_H_ */
