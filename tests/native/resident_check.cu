// A dependent plan beside a kernel that holds 120 of the GPU's SMs: it has to
// end while that kernel still runs, with the results it has on an empty GPU.
// The holder ends by itself after 8 seconds.
#include <cuda_runtime.h>

#include <chrono>
#include <cstdio>
#include <vector>

#include "gpumpi.h"
#include "gpumpi/mpi.cuh"

#define CK(x)                                                                          \
    do {                                                                               \
        cudaError_t e_ = (x);                                                          \
        if (e_ != cudaSuccess) {                                                       \
            printf("%s: %s\n", #x, cudaGetErrorString(e_));                            \
            return 2;                                                                  \
        }                                                                              \
    } while (0)
#define GK(x)                                                                          \
    do {                                                                               \
        int r_ = (x);                                                                  \
        if (r_) {                                                                      \
            printf("%s: %d %s\n", #x, r_, gpumpi_last_error());                        \
            return 2;                                                                  \
        }                                                                              \
    } while (0)

__global__ void hold(volatile int* release, volatile int* started) {
    if (threadIdx.x) return;
    if (blockIdx.x == 0) *started = 1;
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do {
        __nanosleep(2000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    } while (!*release && t - t0 < 8000000000ull);
}

static double seconds() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

int main() {
    const int P = 48, calls = 6;
    const size_t n = 20000;
    double* buf[2];
    std::vector<void*> at[2];
    for (int k = 0; k < 2; k++) {
        CK(cudaMalloc(&buf[k], P * n * 8));
        for (int r = 0; r < P; r++) at[k].push_back(buf[k] + r * n);
    }
    std::vector<double> in(P * n), want(P * n), got(P * n);
    for (size_t i = 0; i < P * n; i++) in[i] = (double)((i * 2654435761u) % 1000) / 1000 - 0.5;
    gpumpi_comm_t comm;
    GK(gpumpi_comm_create(P, &comm));
    std::vector<gpumpi_coll_desc> d(calls);
    for (int i = 0; i < calls; i++)
        d[i] = {comm, GPUMPI_COLL_ALLREDUCE, MPI_DOUBLE, GPUMPI_OP_SUM, 0, n, at[i % 2].data(), at[1 - i % 2].data(), 0, 0};
    gpumpi_plan_t plan;
    GK(gpumpi_plan_create(d.data(), calls, 64, 1, &plan));
    cudaStream_t st, hs;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&hs, cudaStreamNonBlocking));
    volatile int* flags;
    CK(cudaHostAlloc((void**)&flags, 2 * sizeof(int), cudaHostAllocMapped));
    flags[0] = flags[1] = 0;
    CK(cudaFuncSetAttribute(hold, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    bool beside = false;
    for (int k = 0; k < 2; k++) {
        CK(cudaMemcpyAsync(buf[0], in.data(), P * n * 8, cudaMemcpyHostToDevice, st));
        CK(cudaStreamSynchronize(st));
        if (k == 1) {
            hold<<<120, 64, 200 * 1024, hs>>>(flags, flags + 1);
            CK(cudaGetLastError());
            for (double t = seconds(); !flags[1] && seconds() - t < 5;) {
            }
        }
        GK(gpumpi_plan_launch(plan, st));
        if (k == 1) {
            for (double t = seconds(); !beside && seconds() - t < 4;) beside = cudaStreamQuery(st) == cudaSuccess;
            flags[0] = 1;
        }
        CK(cudaStreamSynchronize(st));
        CK(cudaMemcpyAsync((k ? got : want).data(), buf[calls % 2], P * n * 8, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    CK(cudaStreamSynchronize(hs));
    const bool started = flags[1] != 0;
    GK(gpumpi_api_status(nullptr, 0));
    GK(gpumpi_plan_destroy(plan));
    GK(gpumpi_comm_destroy(comm));
    printf("started %d beside %d same %d\n", started, beside, got == want);
    return !(started && beside && got == want);
}
