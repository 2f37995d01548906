// A cluster of two CTAs in which the first gives up a wait for bytes that nobody
// sends, after 64 tries: what each CTA knows of it before and after a sum over
// the group, and the sum.  out[8 * rank + ...]
#include "resident.cuh"

namespace {
constexpr int NT = 256;

__global__ void __launch_bounds__(NT) k_wait(int wait_rank, double* out) {
    using namespace cpdlp;
    __shared__ double sh[res_sh<2, NT / 32>()];
    __shared__ ResWait W;
    const int rank = res_rank<2>();
    int phase = 0;
    unsigned parity = 0;
    if (threadIdx.x == 0) res_wait_init(W);
    res_sync<2>();
    for (int round = 0; round < 2; round++) {
        if (rank == wait_rank) res_receive<2>(W, 0, 16u, parity, 64);
        __syncthreads();
        if (threadIdx.x == 0) out[8 * rank + 4 * round] = W.failed;
        double v[5] = {1.0, 2.0, 3.0, 4.0, 5.0};
        res_sum<5, 2, NT / 32>(v, sh, phase, W);
        if (threadIdx.x == 0) {
            out[8 * rank + 4 * round + 1] = W.failed;
            out[8 * rank + 4 * round + 2] = v[0];
            out[8 * rank + 4 * round + 3] = v[4];
        }
    }
    res_sync<2>();
}
}  // namespace

// 0, or the CUDA error
extern "C" int resident_wait(int wait_rank, double* host_out) {
    double* out = nullptr;
    cudaError_t e = cudaMalloc(&out, 16 * sizeof(double));
    if (e != cudaSuccess) return (int)e;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(NT);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, k_wait, wait_rank, out);
    if (e == cudaSuccess) e = cudaMemcpy(host_out, out, 16 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(out);
    return (int)e;
}
