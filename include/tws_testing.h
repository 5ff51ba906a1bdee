/* tws_testing.h -- test-only entry points of libtws.so.
 *
 * Not part of the drop-in interface (include/tws.h): an integrator has no use
 * for these, and including this header is a deliberate choice.  Nothing here
 * has a counterpart in the reference, whose shaders have no waits that can
 * run out.
 */
#ifndef TWS_TESTING_H
#define TWS_TESTING_H

#include "tws.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Failure-detection hook.  With drop = 1 every tile load of this grid's step
 * kernels arms its barrier for the tile's bytes but issues no copy, and the
 * tiles of the mesh kernel send their neighbours nothing, so each
 * bounded wait (tws_set_wait_limit) runs out with nothing in flight: the
 * kernel records the time-out and returns, and the next tws_sync or
 * tws_batch_sync reports TWS_ERR_TIMEOUT once.  drop = 0 turns it off.
 * Returns TWS_ERR_INVALID for other values. */
TWS_API int tws_test_drop_tile_loads(tws_grid* grid, int drop);

/* With refuse = 1 every launch of the mesh kernel (see tws_step) for this grid
 * fails as one that is too large for its stream's SMs does
 * (cudaErrorCooperativeLaunchTooLarge), before anything is launched: the calls
 * run as the kernel variants.  refuse = 0 turns it off; TWS_ERR_INVALID for
 * other values. */
TWS_API int tws_test_refuse_mesh(tws_grid* grid, int refuse);

/* The packed division of the step kernels, q[i] = d[i] / t[i] for device arrays of
 * n floats (n even), on `stream` (NULL: the legacy default).  Asynchronous. */
TWS_API int tws_test_divide(const float* d, const float* t, float* q, long long n, void* stream);

/* Bytes of the mesh kernel's workspace on the current device now (0: no grid
 * holds one). */
TWS_API size_t tws_test_mesh_workspace(void);

#ifdef __cplusplus
}
#endif

#endif /* TWS_TESTING_H */
