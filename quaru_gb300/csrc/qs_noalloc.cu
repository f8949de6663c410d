// qs_noalloc.cu — measurement probabilities for callers that cannot allocate device memory.
//
// Some callers of this library cannot call cudaMalloc: code that runs while a
// framework owns every byte of device memory through its own allocator, code
// on a latency-critical path where an allocation (and the implicit
// synchronisation it can bring) is not acceptable, or code that must stay
// within a fixed, pre-planned memory budget. They hold their state vector in
// a buffer they allocated themselves and need the probability sums of
// Register::try_measure (src/register.rs:303-315) for it.
//
// qs_measure_probabilities_noalloc() computes them with no allocation of any
// kind: the per-block partial sums go to the file-scope array below, which
// the CUDA module holds on every GPU that loads this library until the
// process exits. The kernels are those of qs_measure_probabilities(), so both give the same sums.
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "qs_kernels.h"

namespace qs {
namespace {

constexpr int kNaMaxBlocks = 4096;  // scratch capacity: 2 doubles per block, 64 KiB in total
constexpr int kNaMaxDevices = 64;

// The scratch: written by every call, read by the same call's final kernel.
// Calls that overlap on the GPU (different streams, or host threads racing)
// share it and race; callers serialise them.
static __device__ __align__(256) double g_noalloc_partials[2 * kNaMaxBlocks];

// Device address of g_noalloc_partials, looked up once per device.
void* g_scratch_addr[kNaMaxDevices] = {nullptr};
std::mutex g_scratch_mu;

int na_err(int code, const std::string& msg) {
    set_last_error_message(msg);
    return code;
}

// Set-up, once per device, with that device current: the host-side name of
// g_noalloc_partials is only a stand-in, so look up its device address. The
// address is kept for the life of the process; cudaDeviceReset (or any other
// teardown of the device's primary context) unloads the module and makes it
// stale, so callers do not reset a device they keep using this entry point on.
int scratch_for_current_device(void** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return na_err(QS_CUDA_ERROR, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
    if (dev < 0 || dev >= kNaMaxDevices) return na_err(QS_INVALID_ARGUMENT, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_partials);
        if (e != cudaSuccess || !p)
            return na_err(QS_CUDA_ERROR, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_scratch_addr[dev] = p;
    }
    *out = g_scratch_addr[dev];
    return QS_OK;
}

}  // namespace
}  // namespace qs

extern "C" int qs_measure_probabilities_noalloc(const void* state, size_t n, int precision, size_t target,
                                                double* out, void* stream, size_t* err) {
    using namespace qs;
    if (!state || !out) return na_err(QS_INVALID_ARGUMENT, "state and out must be device pointers");
    if (precision != QS_PREC_C128 && precision != QS_PREC_C64) return na_err(QS_INVALID_ARGUMENT, "unknown precision");
    // The kernels load whole amplitudes (16 or 8 bytes) and store doubles: a misaligned pointer
    // would fault on the GPU and end the caller's context, so it is refused here instead.
    const uintptr_t amp_align = precision == QS_PREC_C128 ? 16 : 8;
    if (reinterpret_cast<uintptr_t>(state) % amp_align != 0 || reinterpret_cast<uintptr_t>(out) % 8 != 0)
        return na_err(QS_INVALID_ARGUMENT, "state must be aligned to its amplitude size and out to 8 bytes");
    if (n < 1 || n > 40) return na_err(QS_INVALID_ARGUMENT, "n must be in 1..40");
    if (target >= n) {
        if (err) err[0] = target;
        return na_err(QS_INVALID_TARGET, "InvalidTarget(" + std::to_string(target) + ")");
    }
    int dev = 0, sms = 1;
    if (cudaGetDevice(&dev) != cudaSuccess) return na_err(QS_CUDA_ERROR, "cudaGetDevice failed");
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    void* scratch = nullptr;
    int rc = scratch_for_current_device(&scratch);
    if (rc) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const cudaError_t e = launch_measure_probs(state, int(n), precision, int(target), static_cast<double*>(scratch),
                                               kNaMaxBlocks, out, s, sms);
    if (e != cudaSuccess) return na_err(QS_CUDA_ERROR, std::string("launch: ") + cudaGetErrorString(e));
    return QS_OK;
}
