// Internal helpers shared by the libbbpd translation units (not part of the ABI).
#pragma once

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>

#include "bbpd.h"

namespace bbpd {

// Record a message for bbpd_last_error() on this thread and return `code`.
int fail(int code, const char *fmt, ...);
void clear_error();

}  // namespace bbpd

#ifdef __CUDACC__
#include <cuda_runtime.h>

#define BBPD_CUDA_TRY(expr)                                                        \
    do {                                                                           \
        cudaError_t e_ = (expr);                                                   \
        if (e_ != cudaSuccess)                                                     \
            return bbpd::fail(e_ == cudaErrorMemoryAllocation ? BBPD_ERR_OOM      \
                                                              : BBPD_ERR_CUDA,    \
                              "%s: %s (%s:%d)", #expr, cudaGetErrorString(e_),     \
                              __FILE__, __LINE__);                                 \
    } while (0)

namespace bbpd {
// Fails with BBPD_ERR_NO_DEVICE when no CUDA device is visible: this library
// has no CPU implementation to fall back to.
int require_device();
// Stream-ordered temporaries from a pool of the library's own on the current
// device (freed with cudaFreeAsync). The default pool gives everything back to
// the driver at each synchronisation, so a call that ends with one mapped its
// temporaries anew every time; this pool keeps up to kScratchKeep bytes until
// release_scratch (bbpd_release_mirrors) or process exit. Where the default pool
// keeps that much already, the temporaries come from there.
constexpr uint64_t kScratchKeep = (uint64_t)256 << 20;
cudaError_t scratch_malloc(void **p, size_t bytes, cudaStream_t st);
void release_scratch();
inline cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }
}  // namespace bbpd
#endif
