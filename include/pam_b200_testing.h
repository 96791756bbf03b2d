/* pam_b200 -- hooks for the test suite.  NOT part of the product ABI: nothing in the package's
 * hot path calls these, and a host application should not either. */
#ifndef PAM_B200_TESTING_H
#define PAM_B200_TESTING_H

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Forces the CTA tile of the matrix-product kernels so that tests can run every tile shape on the
 * same problem and check that results do not depend on the tile (the library normally picks a
 * 128x128, a 64x64 or, for small or ragged-edged products, a 32x32 tile per problem from a cost
 * model).  0 = by cost model (default), 1 = always 128x128, 2 = always 64x64, 3 = always
 * 32x32 (products that have no 32x32 kernel use 64x64), 4 = 112x128 for plain PAM products whose operands
 * allow it (A contiguous along K, 128-bit loads), else 128x128, 5 = 56x64 for unsplit PAM products whose operands
 * allow it (A contiguous along K, or no 128-bit loads), else 64x64.  Process-wide and not thread-safe, which is
 * why it is kept out of pam_b200.h.  No counterpart in the reference. */
int pamk_test_set_tile_policy(int policy);

/* The tile edge (128, 64 or 32) the cost model gives the PAM product of these dimensions under the
 * current policy, with the automatic split: lets a test pin the measured-best choices without a GPU.
 * Negative (PAMK_ERR_ARG) for an empty problem.  No counterpart in the reference. */
int pamk_test_planned_tile(int64_t batch, int64_t M, int64_t N, int64_t K);

/* Rows per tile (128, 112, 64 or 32) of a plain PAM product of these dimensions and K ranges (0 = the library's choice)
 * whose operands allow every tile, as planned: A contiguous along K, 128-bit loads.  Negative (PAMK_ERR_ARG) for an empty problem or a
 * negative split.  No counterpart in the reference. */
int pamk_test_planned_rows(int64_t M, int64_t N, int64_t K, int split_k);

/* The same for a product in several K ranges as it is launched: ranges planned for 128 rows may run on tiles of 112, with
 * the same bounds.  No counterpart in the reference. */
int pamk_test_split_rows(int64_t M, int64_t N, int64_t K, int split_k);

/* Rows per tile (128, 64, 56 or 32) of an unsplit PAM product as planned, in place, whose A lies contiguous along K or not and whose operands allow
 * 128-bit loads or not.  Negative (PAMK_ERR_ARG) for an empty problem.  No counterpart in the reference. */
int pamk_test_small_rows(int64_t batch, int64_t M, int64_t N, int64_t K, int a_along_k, int wide_loads);

/* Whether PAM products of large tiles run on packed operands: 0 = where it pays (default), 1 = wherever the scratch suffices,
 * 2 = never.  Process-wide and not thread-safe.  No counterpart in the reference. */
int pamk_test_set_packing_policy(int policy);

/* In how many CTAs a wait has run out on the current device since the library was loaded (see pamk_matmul_scratch_bytes):
 * 0 unless something is wrong.  Synchronises.  No counterpart in the reference. */
int pamk_test_expired_waits(unsigned* count);

/* Lets a wait of those kernels run out after `ms` (at most 1000): one CTA of eight warps whose barriers nothing arrives at, the first with that
 * limit.  out, ten values on the device: whether each warp's barrier was reached, the milliseconds until all warps had left, and
 * how many ran out by themselves.  Not counted by pamk_test_expired_waits.  No counterpart in the reference. */
int pamk_test_run_out(unsigned ms, unsigned* out, void* stream);

#ifdef __cplusplus
}
#endif
#endif
