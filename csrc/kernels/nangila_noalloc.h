/* Entry points of libnangila_kernels.so that never allocate.
 *
 * Who this is for: code that wants a checksum of a device buffer but is not in a position to get
 * scratch memory for it — a plugin running inside somebody else's process under a "no allocations
 * after start-up" rule, a callback on a thread where cudaMalloc would deadlock with the caller's own
 * allocator lock, a library that was handed a fixed memory budget it has already spent. The kernel
 * needs no memory beyond the result word.
 *
 * This header has no counterpart in the reference implementation.
 */
#pragma once
#include <cuda_runtime_api.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Largest buffer nangila_crc32_noalloc() accepts: 64 MiB. */
int64_t nangila_crc32_noalloc_max_bytes(void);

/* IEEE CRC32 (the zlib one) of `nbytes` bytes at device address `data`, written to the device word
 * `*out`; queued on `stream`, returns a cudaError_t value (0 = queued). Same result as nangila_crc32().
 *
 * - Calls no cudaMalloc / cudaFree / allocating library routine, and does not synchronize.
 * - nbytes > nangila_crc32_noalloc_max_bytes() is refused with cudaErrorInvalidValue (nothing queued).
 * - Nothing is shared between calls: calls on different streams may overlap as long as their result
 *   words differ. `*out` holds the result only when everything the call queued has run. */
int nangila_crc32_noalloc(const void* data, int64_t nbytes, uint32_t* out, cudaStream_t stream);

#ifdef __cplusplus
}
#endif
