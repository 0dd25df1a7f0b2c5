// Runtime hooks used only by generated kernel modules (not part of the public C ABI).
#pragma once
#include "xgrid_gb300.h"

#ifdef __cplusplus
extern "C" {
#endif

/* While `on` is nonzero on the calling thread, the runtime refuses to allocate
 * device memory for boundary-mask tables and reports an error instead.  The
 * no-alloc entry points of generated modules set it around their call. */
void xg_internal_noalloc_scope(int on);

/* 0 while a call on `stream` may not build boundary-mask tables: inside the scope
 * above, and while the stream is being captured. */
int xg_internal_may_build(void* stream);

/* 1 when the box tables of (core, halo) and of every mask value listed are built. */
int xg_internal_boxes_built(const xg_mask* mask, const int32_t* core, const int32_t* halo, int nvalues,
                            const int32_t* values);

/* Called by an entry whose one launch is short (about 12 us on the GPU at most): xg_call
 * then replays its graph, the cheaper call on the host, instead of launching directly,
 * which leaves a shorter gap on the GPU. */
void xg_internal_short_launch(void);

#ifdef __cplusplus
}
#endif
