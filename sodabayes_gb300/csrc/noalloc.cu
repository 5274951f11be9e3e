// noalloc.cu — genomic values pred = mu + X * effects without any allocation.
//
// Some hosts cannot let this library allocate device memory: a Fortran or C
// host that already owns the GPU through its own memory pool (CUDA Fortran /
// OpenACC runtimes, frameworks with caching allocators), or a latency-bound
// loop that must not pay cudaMalloc/cudaFree and the device-wide
// synchronisation they can imply.  For them sodagpu_compute_dgv_noalloc
// computes the same values as compute_dgv (utilities.f90:616-622, with the
// centring of xscale, utilities.f90:545-552) from device buffers the caller
// owns, using as scratch only the fixed array below.
//
// The scratch is a file-scope __device__ array of SODAGPU_NOALLOC_SCRATCH
// doubles (16 MiB): every GPU that loads this library keeps it until the
// process exits.  Host code cannot use the array's name as a device address,
// so the first call on each device looks the address up with
// cudaGetSymbolAddress (with that device current) and caches it; later calls
// reuse it.  Every call shares the one array: calls that overlap on the GPU
// (different streams, or different host threads on the same device) race on
// it and must be serialised by the caller.  cudaDeviceReset destroys the
// context that holds the array; the cached address is then stale, so a host
// that resets a device must not call this entry point on it again in the
// same process.
//
// The columns are summed in the splits of dgv_splits (dgv.cuh), the same as
// sodagpu_predict's while nind times their number fits the scratch, and in
// fewer above that: the last bits of the result can differ then.  Codes
// outside 0..2 count as 1, the value load_geno gives a missing call
// (utilities.f90:446-449); sodagpu_predict rejects them instead.
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "../../include/sodagpu.h"
#include "dgv.cuh"

namespace {

constexpr int kMaxDevices = 64;

static __device__ __align__(256) double g_dgv_scratch[SODAGPU_NOALLOC_SCRATCH];

std::mutex g_scratch_mu;
double *g_scratch_ptr[kMaxDevices];   // device address per device, 0 until looked up

}  // namespace

extern "C" int sodagpu_compute_dgv_noalloc(int32_t nind, int32_t nloci, const int8_t *codes, int32_t ldg,
                                           const double *freq, double mu, const double *effects, double *pred,
                                           void *stream)
{
    if (nind < 1 || nloci < 1 || ldg < nind || !codes || !freq || !effects || !pred) return SODAGPU_E_ARG;
    if ((int64_t)nind > (int64_t)SODAGPU_NOALLOC_SCRATCH) return SODAGPU_E_ARG;   // beyond the scratch maximum
    int nsplit = soda::dgv_splits(nind, nloci);
    if ((int64_t)nsplit * nind > (int64_t)SODAGPU_NOALLOC_SCRATCH)
        nsplit = (int)((int64_t)SODAGPU_NOALLOC_SCRATCH / nind);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return SODAGPU_E_NODEVICE;
    }
    if (dev < 0 || dev >= kMaxDevices) return SODAGPU_E_UNSUPPORTED;
    double *scratch = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        if (!g_scratch_ptr[dev]) {
            void *ptr = nullptr;
            const cudaError_t e = cudaGetSymbolAddress(&ptr, g_dgv_scratch);
            if (e != cudaSuccess || !ptr) {
                cudaGetLastError();
                return SODAGPU_E_CUDA;
            }
            g_scratch_ptr[dev] = (double *)ptr;
        }
        scratch = g_scratch_ptr[dev];
    }
    if (soda::dgv_enqueue<soda::DGV_RAW>(reinterpret_cast<const uint8_t *>(codes), (size_t)ldg, nullptr, freq, nullptr,
                                         effects, nind, nloci, mu, scratch, (size_t)nind, nsplit, pred,
                                         (cudaStream_t)stream) != cudaSuccess) {
        cudaGetLastError();
        return SODAGPU_E_CUDA;
    }
    return 0;
}
