// Entry points of the translation units that hold the shape-specialised kernels; called by the
// executor in bfly_kernels.cu.
#pragma once
#include <cuda_runtime.h>

#include <cuda.h>

#include "bfly_bw3.h"
#include "bfly_fw2.h"
#include "bfly_mma.h"

namespace bfly {

// Launch the packed-pair forward kernel (after the small kernel that re-orders the twiddles into
// p.packed).  Returns BFLY_OK, a negative status, or kFw2Declined when a tensor cannot be
// described to the TMA unit (the caller then runs the generic kernel).
// `ctas_per_sm`: 1 or 2 (rows per thread up to 14 or 7).  `err`: device address of the flag that a
// kernel whose bounded wait ran out raises.  `launches`: kernels launched.
int fw2_launch(const Fw2Params& p, int ctas_per_sm, int sms, cudaStream_t stream, int* err, int* launches);

// `guard`, here and below: null, or the kernel does nothing while *guard is 0.
// out[b, f] += bias[f], f < len, on a (B, width) matrix with row pitch `pitch` (elements).
int bias_add_launch(float* out, const float* bias, int64_t B, int len, int64_t pitch, const int* guard, int sms, cudaStream_t stream);

// out[c] = sum of g[b, c] over the rows of a (B, cols) matrix with row pitch `pitch`, in an order that B and cols fix.
// `partial`: column_sum_slices(B, cols).floats floats of scratch (bfly_driver.h).  `launches`: kernels launched.
int column_sums_launch(const float* g, int64_t pitch, int64_t B, int cols, float* out, float* partial, const int* guard, cudaStream_t stream, int* launches);
// out[b, c] = sum of g[b, s, c] over s; g (B, S, n), out (B, cols), cols <= n.
int stack_sums_launch(const float* g, int64_t B, int S, int64_t n, int cols, float* out, const int* guard, int sms, cudaStream_t stream);
// rows times width bytes of zeros, rows `pitch` bytes apart (multiples of four), if *guard is not 0 by then.
int guarded_zero_launch(void* p, size_t pitch, size_t width, size_t rows, const int* guard, int sms, cudaStream_t stream);

// Launch the packed-pair backward phase kernel.  The three descriptors (activation in, gradient
// in, gradient out) describe boxes of kBw3Rows rows of the phase's panel (bfly_tma.h).
int bw3_launch(const Bw3Params& p, const CUtensorMap& mx, const CUtensorMap& mg, const CUtensorMap& mo, cudaStream_t stream,
               int* err);

// The kernels of bfly_mma.h.  `err` as for fw2_launch.
int mma_prep_launch(const MmaPrep& p, bool cplx, cudaStream_t stream);
int mma_fw_launch(const MmaPass& p, int sms, cudaStream_t stream, int* err);
int mma_bw_launch(const MmaPass& p, int ctas, cudaStream_t stream, int* err);
int mma_post_launch(const MmaPost& p, bool cplx, cudaStream_t stream, int* launches);

// Adds to the count that bfly_launch_count reports (kernels launched by the other translation units).
void count_launches(int n);

}  // namespace bfly
