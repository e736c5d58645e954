// Self-tests of what the kernels rely on and no solve can show.
//
// Bounded waits of every persistent kernel of the library.  Each case runs one
// wait whose condition nothing ever makes true -- a grid barrier that counts one
// block more than the launch has, a counter barrier with an unreachable target,
// an mbarrier no one arrives at, a record or a report no one writes -- and
// records whether the wait gave up after its time limit and raised its error
// flag, as it must for a solver kernel to return TSE_STATUS_BARRIER_TIMEOUT
// instead of holding the GPU.  Nothing faults: the kernels only wait, give up
// and return.
#include "tse_dc.cuh"
#include "tse_quotient.cuh"
#include "tse_resident.cuh"

namespace tse {

// result[which]: 1 = the wait returned false with its error flag raised
__global__ void __launch_bounds__(128) selftest_wait_kernel(int which, GridBarrier* bar,
                                                            unsigned* counter, int* result,
                                                            unsigned long long timeout_ns) {
    if (which == 0) {
        const bool ok = grid_sync(bar, gridDim.x + 1, timeout_ns);
        if (blockIdx.x == 0 && threadIdx.x == 0)
            result[0] = (!ok && *(volatile int*)&bar->error) ? 1 : 0;
    } else if (which == 1) {
        const bool ok = count_sync(counter, gridDim.x + 1, bar, timeout_ns);
        if (blockIdx.x == 0 && threadIdx.x == 0)
            result[1] = (!ok && *(volatile int*)&bar->error) ? 1 : 0;
    } else {
        __shared__ __align__(8) uint64_t mb;
        __shared__ int err;
        if (threadIdx.x == 0) {
            mbar_init(&mb, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            err = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const bool ok = mbar_wait_flag(&mb, 0u, (volatile int*)&err, timeout_ns);
            // complete the phase no one completed, so the barrier is left idle
            mbar_arrive(&mb);
            result[2] = (!ok && err) ? 1 : 0;
        }
        __syncthreads();
    }
}

// The resident solves' waits: an edge record and a sum record nobody writes
// (result[0], result[1]: gave up, flags raised), and a solve that one block
// leaves early.  There block 1's edge wait runs out; it still makes its partial
// sum and leaves.  Block 0, late, finds that sum and knows of nothing
// (result[2]: its sum is good); the last block to leave does (result[3]).
__global__ void __launch_bounds__(kResMaxThreads) selftest_resident_kernel(int which, GridBarrier* bar,
                                                                           unsigned* counter, uint64_t* words,
                                                                           int* result,
                                                                           unsigned long long timeout_ns) {
    __shared__ ResSumShared sum;
    __shared__ uint4 ring[1];
    __shared__ int hrec[1], s_err;
    __shared__ unsigned short hp[1];
    volatile int* err = &s_err;
    uint64_t* slots = words + 4;   // words 0 .. 3: one edge record, never written
    if (threadIdx.x == 0) {
        s_err = 0;
        hrec[0] = 0;
        hp[0] = 0;
    }
    __syncthreads();
    if (which == 0) {
        res_poll<kResMaxThreads>(words, 2, 1u, ring, hrec, hp, 1, bar, err, timeout_ns);
        __syncthreads();
        if (threadIdx.x == 0) result[0] = *err && *(volatile int*)&bar->error;
    } else if (which == 1) {
        if (threadIdx.x == 0) {
            double A = 0.0, B = 0.0;
            const bool ok = res_poll_pair(slots, 1u, A, B, bar, err, timeout_ns);
            result[1] = !ok && *err && *(volatile int*)&bar->error;
        }
    } else {
        const unsigned b = blockIdx.x;
        if (b == 1) {
            res_poll<kResMaxThreads>(words, 2, 1u, ring, hrec, hp, 1, bar, err, timeout_ns);
        } else if (threadIdx.x == 0) {
            const uint64_t t0 = globaltimer();
            while (globaltimer() - t0 < 2 * timeout_ns) __nanosleep(1000);
        }
        __syncthreads();
        double u = 1.0, v = 1.0;
        const bool ok = res_team_sum<kResMaxThreads, RES_GRID>(u, v, sum, slots, 2u, b, 0u, bar, err, timeout_ns);
        if (b == 0 && threadIdx.x == 0) result[2] = ok && u == 2.0 * kResMaxThreads;
        bool failed = !ok;
        if (res_last<RES_GRID>(counter, 2u, b, failed)) result[3] = failed;
    }
}

// The staged sweep's wait for other blocks' reports
__global__ void selftest_report_kernel(GridBarrier* bar, unsigned* counter, int* result,
                                       unsigned long long timeout_ns) {
    __shared__ int s_err;
    s_err = 0;
    const bool ok = seg_wait(counter, 1u, bar, (volatile int*)&s_err, timeout_ns);
    *result = !ok && s_err && *(volatile int*)&bar->error;
}

// The flux kernels' quotients and reciprocals, for a comparison with divisions
__global__ void selftest_quotient_kernel(const double* a, const double* b, double* q, double* y, long long n) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const Divisor d = divisor(b[t]);
    q[t] = quotient_0(a[t], d);
    y[t] = d.y;
}

}  // namespace tse

using namespace tse;

extern "C" int32_t tse_selftest_bounded_waits(int32_t* d_result, double timeout_s, void* d_ws,
                                              size_t ws_bytes, void* stream_) {
    if (!d_result || !d_ws || ws_bytes < 512 || !(timeout_s > 0.0)) return TSE_ERR_ARG;
    if (timeout_s > 5.0) timeout_s = 5.0;
    const unsigned long long ns = (unsigned long long)(timeout_s * 1e9);
    cudaStream_t stream = (cudaStream_t)stream_;
    GridBarrier* bar = (GridBarrier*)d_ws;
    unsigned* counter = (unsigned*)((char*)d_ws + 256);
    int* result = (int*)d_result;
    if (cudaMemsetAsync(d_result, 0, 3 * sizeof(int32_t), stream) != cudaSuccess) return TSE_ERR_LAUNCH;
    for (int which = 0; which < 3; ++which) {
        if (cudaMemsetAsync(d_ws, 0, 512, stream) != cudaSuccess) return TSE_ERR_LAUNCH;
        // the two blocks of the barrier cases wait on each other: co-resident
        // by a cooperative launch
        int w = which;
        void* args[] = {(void*)&w, (void*)&bar, (void*)&counter, (void*)&result, (void*)&ns};
        const cudaError_t e =
            which < 2 ? cudaLaunchCooperativeKernel((const void*)selftest_wait_kernel, dim3(2), dim3(128),
                                                    args, 0, stream)
                      : cudaLaunchKernel((const void*)selftest_wait_kernel, dim3(1), dim3(128), args, 0,
                                         stream);
        if (e != cudaSuccess) return TSE_ERR_LAUNCH;
    }
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

extern "C" int32_t tse_selftest_resident_waits(int32_t* d_result, double timeout_s, void* d_ws, size_t ws_bytes,
                                               void* stream_) {
    const size_t words = 4 * sizeof(uint64_t) + kResSlotBytes, need = 512 + words;
    if (!d_result || !d_ws || ws_bytes < need || !(timeout_s > 0.0)) return TSE_ERR_ARG;
    if (timeout_s > 1.0) timeout_s = 1.0;
    unsigned long long ns = (unsigned long long)(timeout_s * 1e9);
    cudaStream_t stream = (cudaStream_t)stream_;
    GridBarrier* bar = (GridBarrier*)d_ws;
    unsigned* counter = (unsigned*)((char*)d_ws + 256);
    uint64_t* w = (uint64_t*)((char*)d_ws + 512);
    int* result = (int*)d_result;
    if (cudaMemsetAsync(d_result, 0, 5 * sizeof(int32_t), stream) != cudaSuccess) return TSE_ERR_LAUNCH;
    for (int which = 0; which < 4; ++which) {
        if (cudaMemsetAsync(d_ws, 0, need, stream) != cudaSuccess) return TSE_ERR_LAUNCH;
        if (which == 3) {
            selftest_report_kernel<<<1, 1, 0, stream>>>(bar, counter, result + 4, ns);
            continue;
        }
        void* args[] = {(void*)&which, (void*)&bar, (void*)&counter, (void*)&w, (void*)&result, (void*)&ns};
        if (cudaLaunchCooperativeKernel((const void*)selftest_resident_kernel, dim3(which == 2 ? 2 : 1),
                                        dim3(kResMaxThreads), args, 0, stream) != cudaSuccess)
            return TSE_ERR_LAUNCH;
    }
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}

extern "C" int32_t tse_selftest_quotients(const double* a, const double* b, double* q, double* y, int64_t n,
                                          void* stream_) {
    if (!a || !b || !q || !y || n < 1 || n > (1LL << 31)) return TSE_ERR_ARG;
    selftest_quotient_kernel<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock, 0, (cudaStream_t)stream_>>>(a, b, q, y,
                                                                                                       n);
    return cudaGetLastError() == cudaSuccess ? TSE_OK : TSE_ERR_LAUNCH;
}
