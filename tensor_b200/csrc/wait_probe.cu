// A kernel whose only job is to let a bounded wait run out (see launch_wait_probe in kernels.h): the way the host learns
// of a kernel that gave up (status word -> OTT_ERR_DEVICE_WAIT at the next ott_sync, word cleared) can then be tested without
// faulting, trapping or hanging anything.
#include "kernels.h"
#include "umma_primitives.cuh"

namespace ottk {

namespace {
__global__ void wait_probe_kernel(uint32_t* status, unsigned long long limit_ns) {
    __shared__ alignas(8) unsigned long long bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        umma::mbar_init(umma::smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // Phase 0 of a freshly initialised barrier with one pending arrival: nobody arrives before lane 0 of the waiting warp has given up
    // (the other lanes have more time). What the others then see, the arrival or the abort flag, must not matter: 0x200 reports a lane
    // that was told to go on.
    volatile int* flag = &abort_flag;
    if (threadIdx.x < 32) {
        const bool ok = umma::mbar_wait_warp(umma::smem_u32(&bar), 0, flag, status, 0x100u, threadIdx.x == 0 ? limit_ns : 4 * limit_ns);
        if (ok) atomicOr(status, 0x200u);
    } else if (threadIdx.x == 32) {
        const unsigned long long t0 = umma::globaltimer_ns();
        while (*flag == 0 && umma::globaltimer_ns() - t0 < 8 * limit_ns) {}
        umma::mbar_arrive(umma::smem_u32(&bar));
    }
    __syncthreads();
}
}  // namespace

cudaError_t launch_wait_probe(cudaStream_t stream, uint32_t* status, unsigned long long limit_ns) {
    wait_probe_kernel<<<1, 64, 0, stream>>>(status, limit_ns);
    return cudaGetLastError();
}

}  // namespace ottk
