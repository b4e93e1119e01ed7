/* b2_local_all_reduce_no_alloc — an all-reduce over buffers that all live on ONE GPU, for callers
 * that must not allocate.
 *
 * This entry point has no counterpart in the reference library (nano-nccl); it is an addition of
 * this project.
 *
 * Who needs it. Some programs that embed this library are not free to call cudaMalloc (or any
 * routine that allocates on their behalf) at the moment they want to reduce something:
 *   - a server that handed every byte of device memory to its own pool at start-up, so that a
 *     later cudaMalloc either fails or takes memory the pool was sized to own;
 *   - a latency-sensitive loop, where cudaMalloc/cudaFree would stall the device behind an
 *     implicit synchronisation at an unpredictable point;
 *   - code that runs under a "no allocation after initialisation" rule (real-time or safety
 *     reviews often impose one).
 * The communicator's own entry points are of no use to them: creating a communicator allocates
 * control blocks, staging memory and events. This function is one launch of the kernel that a
 * communicator uses for ranks that share a GPU (kernels/sm100/local_collectives.cu), which needs no
 * memory but the caller's buffers.
 *
 * What it computes. `nranks` input buffers and `nranks` output buffers of `count` elements, all on
 * the current device. Every output receives the element-wise reduction (sum, avg, max, min; fp32
 * accumulation for fp16/bf16; NaN-propagating max/min) of all inputs. Inputs and outputs must not
 * overlap: any two byte ranges that share a byte (an input with an output, or two outputs) are
 * rejected, as is a count whose byte size overflows size_t. Work is enqueued on `stream`; the call
 * returns without waiting for it.
 *
 * Limits and errors. nranks must be between 1 and B2_NO_ALLOC_MAX_RANKS (8); larger values are
 * rejected with a message (see b2_last_error) and nothing is launched. count must be positive.
 * Return value: 0 on success, 2 for a rejected argument, 1 for a CUDA failure.
 *
 * Sharing. Calls keep nothing between them: any number may run at once, on any streams, and any call
 * may be captured into a graph.
 *
 * `status_record` is accepted for callers of earlier versions, whose kernel had waits that could run
 * out; nothing is written to it.
 */
#pragma once

#include <stddef.h>

#ifdef __cplusplus
extern "C" {
#endif

#define B2_NO_ALLOC_MAX_RANKS 8

/* dtype: 0 float, 1 fp16, 2 bf16. redop: 0 sum, 1 avg, 2 max, 3 min. stream: a cudaStream_t. */
int b2_local_all_reduce_no_alloc(const void* const* inputs, void* const* outputs, int nranks, size_t count, int dtype,
                                 int redop, void* stream, void* status_record);

#ifdef __cplusplus
}
#endif
