// State transfers of ibpm_set_state and ibpm_get_state and the per-call read-back
// of the step, by kernels that read and write page-locked host memory directly.
//
// A copy engine transfer costs several µs to set up, and a state has up to six
// pieces, four of them pitched, which the copy engines write to the device row by
// row; one launch takes all pieces at the link's rate.  A whole state without q0,
// page-locked, copies -> kernel: 64² x 3 levels (0.58 MB) read 40.5 -> 28.5 µs,
// written 131 -> 27; 128² x 5 (3.9 MB) 99 -> 92 and 341 -> 92 µs.  kPackBytes is
// set by the reads: at 200² x 3 (5.7 MB) they take 131 by copies and 126 by the
// kernel, at 256² x 5 (15.7 MB) 308 and 314, and copies leave the SMs free.
#include "host_range.h"
#include "ibpm_internal.cuh"

#include <cuda.h>

namespace ibpm {

namespace {

// Piece blockIdx.y: rows of n1 values, P apart on the device (a Γ-like field),
// contiguous on the host; n1 = P for a contiguous piece.
template <bool TO_DEVICE>
__global__ void __launch_bounds__(256) pack_kernel(const __grid_constant__ PackArgs a) {
    const PackPiece& s = a.piece[blockIdx.y];
    const long long step = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < s.n; t += step) {
        const long long d = s.P == s.n1 ? t : t + t / s.n1 * (s.P - s.n1);
        if constexpr (TO_DEVICE) s.dev[d] = s.host[t];
        else s.host[t] = s.dev[d];
    }
}

__global__ void __launch_bounds__(256) readback_kernel(const double* __restrict__ hist, double* out, int n,
                                                       const int* status, int* status_out) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) out[t] = hist[t];
    if (status_out && threadIdx.x == 0) *status_out = *status;
}

}  // namespace

// The page-locked range of an address, by the driver's query (the runtime's does
// not tell the range), all attributes in one call.
static HostRange host_range(const void* p) {
    using Query = CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
    static const Query query = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPoint("cuPointerGetAttributes", &fn, cudaEnableDefault, &found);
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<Query>(fn) : nullptr;
    }();
    unsigned type = 0, managed = 0;
    CUdeviceptr start = 0, dev = 0;
    size_t size = 0;
    CUpointer_attribute want[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* got[] = {&type, &managed, &dev, &start, &size};
    if (!query || query(5, want, got, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS) return {};
    return {type == CU_MEMORYTYPE_HOST && !managed, static_cast<uintptr_t>(start), size, reinterpret_cast<void*>(dev)};
}

double* locked_host(const double* host, long long n) { return locked_whole(host, n, host_range); }

cudaError_t launch_pack(const PackArgs& a, int npieces, bool to_device, cudaStream_t st) {
    long long most = 0;
    for (int i = 0; i < npieces; ++i) most = a.piece[i].n > most ? a.piece[i].n : most;
    const long long blocks = (most + 1023) / 1024;
    const dim3 grid((unsigned)(blocks < 148 ? blocks : 148), npieces);
    if (to_device) pack_kernel<true><<<grid, 256, 0, st>>>(a);
    else pack_kernel<false><<<grid, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_readback(const double* hist, double* out, int n, const int* status, int* status_out,
                            cudaStream_t st) {
    readback_kernel<<<1, 256, 0, st>>>(hist, out, n, status, status_out);
    return cudaGetLastError();
}

}  // namespace ibpm
