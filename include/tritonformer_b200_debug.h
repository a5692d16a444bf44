/*
 * tritonformer_b200 -- test and tuning switches of the kernel library.  Not part of the operator
 * interface: nothing here has a counterpart in the reference, and a host that only runs the
 * operators never needs this file.
 */
#ifndef TRITONFORMER_B200_DEBUG_H
#define TRITONFORMER_B200_DEBUG_H

#ifdef __cplusplus
extern "C" {
#endif

/* Test and tuning switches.
 *   key 0: value 1 sends every GEMM to the generic-stride kernel.
 *   key 1: value 1 sends every attention call to the mma.sync kernels.
 *   key 2: attention: bit 5 (32) walks the (tile, batch*head) items slice by slice instead of longest first.
 *   key 3: value 1 launches every kernel fully serialised (no programmatic dependent launch: a
 *          kernel's set-up no longer overlaps its predecessor's tail).
 *   key 4: GEMM: bit 0 whole tiles only (no sharing of a tile's contraction between SMs), bit 5 (32)
 *          no persistent CTA-pair kernel, bit 7 (128) no one-wave kernel, bits 16-27 the one plan the one-wave kernel
 *          may use (tfb_debug_gemm_plan).
 *   key 6: how many SMs the persistent GEMM grids leave free (for a collective that runs beside
 *          them on another stream); 0 by default.
 *   key 7: the registers a thread that the attention backward's kernels are taken to have been built with; 0: what they
 *          have.  Where the number does not cover a kernel's split of its registers, the mma.sync kernels take the call.
 * Accepted and without effect, for hosts that still set them: key 5, bits 0, 1, 6 and 7 of key 2, bit 6 of key 4 (they belonged to
 * the cycle counters and to timing experiments of earlier kernels).                                  */
void tfb_debug_set(int key, int value);
/* The kernels count no cycles any more.  Sets out16 to zeros and returns the error code of what is not supported.  */
int tfb_debug_counters(unsigned long long* out16);
/* What the one-wave GEMM kernel does with an M x N x K product (b_mn: B is contiguous along N) under the switches in force:
 * 0 if the product goes to the persistent kernels, else 1 + tile width / 64 * 2 + (on CTA pairs ? 1 : 0) + 16 * the number
 * of workers that share a tile's contraction.                                              */
int tfb_debug_gemm_plan(long long M, long long N, long long K, int b_mn);
/* The width of the tiles that the persistent CTA-pair kernel gives such a product, 0 if it does not get it (a_mn: A is contiguous
 * along M; b_rows_64: the rows of B begin on 64-byte boundaries).                                              */
int tfb_debug_gemm_pair_width(long long M, long long N, long long K, int a_mn, int b_mn, int b_rows_64);
/* Launches a one-warp kernel that takes tensor memory, waits `limit_ns` nanoseconds on an mbarrier
 * that nothing arrives at, gives up, records 0x7e00 in the device status word, frees its tensor memory
 * and returns: the expiry path of the library's bounded waits, without a fault, a trap or an unbounded
 * spin.  waited_ok (device int, may be null) receives 0 when the wait ran out.  Tests only.        */
int tfb_debug_wait_probe(unsigned long long limit_ns, int* waited_ok, void* stream);

#ifdef __cplusplus
}
#endif
#endif
