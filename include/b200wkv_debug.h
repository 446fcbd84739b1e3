/*
 * b200wkv_debug - a schedule query of libb200wkv.so that exists for its tests.  Not part of the
 * boundary a host framework binds (that is b200wkv.h); no jaxrwkv interface corresponds to it.
 * It launches nothing.
 */
#ifndef B200WKV_DEBUG_H_
#define B200WKV_DEBUG_H_

#ifdef __cplusplus
extern "C" {
#endif

/* Decoding (b200wkv7_step_inplace): thread blocks that a full launch puts on an SM, and how many would fit one.  The kernel
 * deals the work out in equal shares, so the two have to be equal.  Needs a device. */
int b200wkv_debug_step_residency(int dtype, int* grid_per_sm, int* fit_per_sm);

#ifdef __cplusplus
}
#endif
#endif  /* B200WKV_DEBUG_H_ */
