/*
 * b200wkv_debug - schedule queries of libb200wkv.so that exist for its tests.  Not part of the
 * boundary a host framework binds (that is b200wkv.h); no jaxrwkv interface corresponds to them.
 * They launch nothing.
 */
#ifndef B200WKV_DEBUG_H_
#define B200WKV_DEBUG_H_

#ifdef __cplusplus
extern "C" {
#endif

/* Decoding (b200wkv7_step_inplace): thread blocks that a full launch puts on an SM, and how many would fit one.  The kernel
 * deals the work out in equal shares, so the two have to be equal.  Needs a device. */
int b200wkv_debug_step_residency(int dtype, int* grid_per_sm, int* fit_per_sm);

/* RWKV-7 forward, bf16, with a workspace: the form that a call takes on a device of `sms` SMs which takes clusters of up to
 * `largest_cluster` thread blocks (a whole B200: 148, 16).  0: the walk, 1: blocks side by side, n > 2: rings of n.  Needs no device. */
int b200wkv_debug_wkv7_fwd_form(int sms, int largest_cluster, int B, int T, int H, int residual);

#ifdef __cplusplus
}
#endif
#endif  /* B200WKV_DEBUG_H_ */
