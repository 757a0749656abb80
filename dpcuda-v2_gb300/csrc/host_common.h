// host_common.h -- error reporting and launch helpers shared by the host-side
// translation units of the library.
#pragma once
#include <cuda_runtime.h>

#include <unistd.h>

#include "../../include/dpg.h"

namespace dpg {
// Records a message for dpg_last_error() (thread-local) and returns `code`.
int set_error(int code, const char *fmt, ...);

// Whether a FIRE minimisation tests its mean energy: against a target, or against
// zero where energies can be negative.
inline int pe_is_read(double pe_target, double pe_diff_target, double e_c, double n_c) {
    return pe_target > 0 || pe_diff_target > 0 || !(e_c > 0) || !(n_c > 0);
}

// cudaMemcpyAsync to the caller's host memory.  Into pages that were not touched
// yet (every array that a caller has just allocated) the driver copies at
// 1.2 GB/s, four arrays of 262144 doubles in 6.7 ms; a byte written to each page
// first makes that 0.3, and costs nothing that shows where the pages are there.
inline cudaError_t copy_out(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    static const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    cudaPointerAttributes a = {};
    if (bytes >= 16 * page) {
        if (cudaPointerGetAttributes(&a, dst) != cudaSuccess) (void)cudaGetLastError();
        else if (a.type == cudaMemoryTypeUnregistered)
            for (size_t k = 0; k < bytes; k += page) static_cast<volatile char *>(dst)[k] = 0;
    }
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
}
}  // namespace dpg

#define DPG_CK(x)                                                                          \
    do {                                                                                   \
        cudaError_t e_ = (x);                                                              \
        if (e_ != cudaSuccess)                                                             \
            return ::dpg::set_error(DPG_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__, #x,  \
                                    cudaGetErrorString(e_));                               \
    } while (0)

#define DPG_TRY(x)                   \
    do {                             \
        int r_ = (x);                \
        if (r_ != DPG_OK) return r_; \
    } while (0)
