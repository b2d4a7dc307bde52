// lsh_probe.cu -- lsh_probe_wait_bound (include/lsh.h): shows on the device
// that the passes' bounded waits give up and report instead of hanging.
//
// Blocks run the waits the library uses between passes on completion counters
// that nothing increments: the first dep_begin (lsh_kernels.cuh: the colour
// passes and the adjoint's) and then queue_wait by one thread (lsh_queue.cuh);
// the others tile_begin (the flux pass's steps), over every tile of a row and
// over the listed ones, and queue_wait by a block's threads, a row each (the
// queues).  Each gives up after its bound (about 2 s of %globaltimer) and
// records it: dep_begin and tile_begin in the time record's error word,
// queue_wait in its abort flag.  The kernel then returns, and the context
// stays usable.

#include <cuda_runtime.h>

#include <string>

#include "../../include/lsh.h"
#include "lsh_kernels.cuh"
#include "lsh_queue.cuh"
#include "lsh_setup.h"

namespace {

constexpr int kRows = 64;  // counters, all zero
constexpr int kWaits = 5;

struct WaitProbe {
    TimeRec tm[3];
    unsigned ctr[kRows];
    int abort_flag[2];
    int listed[3];  // tiles of the rows that block 2 waits for
    int out[kWaits];  // 1 where a wait gave up and left its mark
};

__global__ void k_wait_probe(WaitProbe* w) {
    if (blockIdx.x == 0) {
        Dep d;
        d.wait = w->ctr;  // the wait for 1 never ends by itself
        d.target = 1;
        d.kind = kDepCell;
        d.ntiles = 1;
        dep_begin(d, &w->tm[0], 0, 0);
        if (threadIdx.x == 0) {
            unsigned long long start = 0;
            w->out[1] = queue_wait(w->ctr, 0, 0, 1u, &w->abort_flag[0], start) && w->abort_flag[0];
            w->out[0] = (w->tm[0].err >> LSH_ERR_TIMEOUT) & 1;
        }
    } else if (blockIdx.x < 3) {
        // tile row 1 of 3: waits for the rows 0 to 2
        const int b = (int)blockIdx.x;
        TileMap m{};
        m.ntx = 1;
        m.nty = 3;
        m.count = (b == 2) ? w->listed : nullptr;
        TileDep d;
        d.wait = w->ctr;
        d.per = 2;
        tile_begin(d, m, &w->tm[b], 1, 1);
        if (threadIdx.x == 0) w->out[1 + b] = (w->tm[b].err >> LSH_ERR_TIMEOUT) & 1;
    } else {
        unsigned long long start = 0;
        const bool gave_up = queue_wait(w->ctr, (int)threadIdx.x, kRows - 1, 1u, &w->abort_flag[1], start, (int)blockDim.x);
        const int all = __syncthreads_and(gave_up);
        if (threadIdx.x == 0) w->out[4] = all && w->abort_flag[1];
    }
}

int probe_fail(cudaError_t e, const char* what) {
    lsh::set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
    (void)cudaGetLastError();
    return LSH_ERR_CUDA;
}

}  // namespace

extern "C" int lsh_probe_wait_bound(int device, int* status_out, double* ms_out) {
    if (!status_out) return LSH_ERR_INVALID;
    if (lsh_check_device() != 0) return LSH_ERR_NO_DEVICE;
    if (device >= 0) {
        cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) return probe_fail(e, "cudaSetDevice");
    }
    WaitProbe* w = nullptr;
    cudaError_t e = cudaMalloc(&w, sizeof(WaitProbe));
    if (e != cudaSuccess) return probe_fail(e, "cudaMalloc");
    WaitProbe init{};
    for (int& n : init.listed) n = 1;
    e = cudaMemcpy(w, &init, sizeof(init), cudaMemcpyHostToDevice);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    if (e == cudaSuccess) e = cudaEventRecord(e0);
    if (e == cudaSuccess) {
        k_wait_probe<<<4, 32>>>(w);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaEventRecord(e1);
    if (e == cudaSuccess) e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    WaitProbe res{};
    if (e == cudaSuccess) e = cudaMemcpy(&res, w, sizeof(res), cudaMemcpyDeviceToHost);
    // the device still answers after the waits gave up
    if (e == cudaSuccess) e = cudaMemset(w, 0, sizeof(WaitProbe));
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(w);
    if (e != cudaSuccess) return probe_fail(e, "lsh_probe_wait_bound");
    if (ms_out) *ms_out = ms;
    *status_out = LSH_ERR_TIMEOUT;
    for (int k = 0; k < kWaits; ++k)
        if (!res.out[k]) *status_out = LSH_OK;
    return LSH_OK;
}
