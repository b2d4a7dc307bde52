// TEST INFRASTRUCTURE: the device forms of lsh_ieee.h against CUDA's own
// round-to-nearest division, reciprocal and square root.  Per operand pair,
// one bit for each operation that differs (NaN results count as equal).
#include <cuda_runtime.h>

#include "../../landslidehysea_gb300/csrc/lsh_ieee.h"

namespace {

__device__ int differ(double a, double b) {
    return (__double_as_longlong(a) != __double_as_longlong(b)) && !(a != a && b != b);
}

__global__ void k_check(const double* a, const double* b, long long n, unsigned long long* bad) {
    unsigned long long m = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        m += differ(lshm::div(a[i], b[i]), __ddiv_rn(a[i], b[i]));
        m += differ(lshm::rcp(b[i]), __drcp_rn(b[i]));
        m += differ(lshm::root(a[i]), __dsqrt_rn(a[i]));
        m += differ(lshm::root(fabs(b[i])), __dsqrt_rn(fabs(b[i])));
    }
    if (m) atomicAdd(bad, m);
}

}  // namespace

// Mismatches over n operand pairs, or -1 on a CUDA error.
extern "C" long long ieeec_check_gpu(const double* host_a, const double* host_b, long long n) {
    double* d = nullptr;
    unsigned long long* bad = nullptr;
    long long out = -1;
    if (cudaMalloc(&d, 2 * sizeof(double) * n) != cudaSuccess) return -1;
    if (cudaMalloc(&bad, sizeof(*bad)) == cudaSuccess && cudaMemset(bad, 0, sizeof(*bad)) == cudaSuccess &&
        cudaMemcpy(d, host_a, sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess &&
        cudaMemcpy(d + n, host_b, sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess) {
        k_check<<<1024, 128>>>(d, d + n, n, bad);
        unsigned long long h = 0;
        if (cudaGetLastError() == cudaSuccess && cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost) == cudaSuccess)
            out = (long long)h;
    }
    cudaFree(d);
    cudaFree(bad);
    return out;
}
