// internal.h -- declarations shared by the host planner (api.cpp) and the
// kernel translation units.  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <functional>
#include <string>

#include "../../include/genfft_gb300.h"

namespace gfft {

// thrown inside the library, converted to a status at the C boundary
struct Error {
    gfft_status status;
    std::string msg;
};
[[noreturn]] void fail(gfft_status st, const std::string &msg);
void set_last_error(const char *msg);  // the thread's gfft_last_error() text
void check_cuda(cudaError_t e, const char *what);
// GFFT_ERR_ARCH unless the current device is an sm_103 (GB300)
void check_device();

// ---- fused single-kernel C2C (c2c_fused.cu) ------------------------------
struct FusedC2CArgs {
    const void *in;
    void *out;
    long long batch;
    long long idist, odist;       // elements between transforms
    long long istride, ostride;   // elements between points
    const void *tw;               // device twiddle table for (dtype, logn)
    const void *tw_tma = nullptr; // that of the persistent version, if there is one
    double scale = 1.0;           // applied to every output (norm= scaling)
    bool host = false;            // in / out are host memory the kernel reaches over the link
};
int fused_max_logn(int dtype);
size_t fused_twiddle_count(int dtype, int logn);              // complex elements
void fused_twiddle_fill(int dtype, int logn, void *host_buf);  // writes that many
cudaError_t launch_fused_c2c(int dtype, int logn, int inverse, const FusedC2CArgs &a,
                             cudaStream_t st);

// ---- the persistent versions for fp32, complex lengths 2^12 .. 2^14
// (fused_tma.cu): many transforms of dense, 16-byte aligned input ----------
constexpr int FUSED_TMA_MIN = 12, FUSED_TMA_MAX = 14;
size_t fused_tma_twiddle_count(int logn);
void fused_tma_twiddle_fill(int logn, void *host_buf);
bool fused_tma_takes(int logn, bool real, long long batch);
cudaError_t launch_fused_tma_c2c(int logn, int inverse, const FusedC2CArgs &a, cudaStream_t st);
// C2C of packed transforms: number w is at element off[w], even
cudaError_t launch_fused_tma_at(int logn, int inverse, const void *in, void *out, const long long *off, long long count,
                                const void *tw, cudaStream_t st);
// distances in complex elements; x2 / half: interior bins doubled / halved
cudaError_t launch_fused_tma_r2c(int logh, bool x2, const void *in, void *out, long long batch, long long idist,
                                 long long odist, const void *tw, const void *dtw, cudaStream_t st, double scale);
cudaError_t launch_fused_tma_c2r(int logh, bool half, const void *in, void *out, long long batch, long long idist,
                                 long long odist, const void *tw, const void *dtw, cudaStream_t st, double scale);

// Opts fn in to `smem` bytes of dynamic shared memory when that is above
// the 48 KB default, once per (device, function).
cudaError_t ensure_smem(const void *fn, size_t smem);

// Launches fn as a programmatic dependent of the previous kernel on the
// stream: its CTAs may start while that kernel's last wave drains, and the
// kernel (which begins with pdl_enter()) waits for that kernel's completion
// before it touches global memory.  GFFT_PDL=0: an ordinary launch.
cudaError_t launch_pdl(const void *fn, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t st);

// ---- device twiddle cache (api.cpp) --------------------------------------
// Returns a device pointer to the table made by `fill` (count complex
// elements of dtype), cached per (device, key) for the process lifetime.
const void *cached_table(const std::string &key, int dtype, size_t count,
                         const std::function<void(void *)> &fill);

}  // namespace gfft
