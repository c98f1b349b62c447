// Sums of 32 values by the solvers' warp_sum, a warp per sum (built and called by test_gpu_warp_sums.py).
#include "../../poissonrecon_gpu_gb300/csrc/cg_common.cuh"

using namespace prgpu;

__global__ void k_doubles(const double* v, int n, double* out) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    const double s = warp_sum(v[32 * w + lane]);
    if (__shfl_sync(0xffffffffu, s, 31) != s && s == s) out[w] = INFINITY;   // every lane gets the sum
    else if (lane == 0) out[w] = s;
}
__global__ void k_pairs(const float2* v, int n, double* out) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    FSum f;
    f.h = v[32 * w + lane].x;
    f.l = v[32 * w + lane].y;
    const double s = warp_sum(f);
    if (lane == 0) out[w] = s;
}

// in: n x 32 doubles, or pairs of floats when 'pairs'; host arrays
extern "C" int warp_sums(const void* in, int n, int pairs, double* out) {
    void* d = nullptr;
    double* o = nullptr;
    if (cudaMalloc(&d, (size_t)n * 256) || cudaMalloc(&o, (size_t)n * 8)) return 1;
    if (cudaMemcpy(d, in, (size_t)n * 256, cudaMemcpyHostToDevice)) return 1;
    const int blocks = (n + 3) / 4;
    if (pairs) k_pairs<<<blocks, 128>>>((const float2*)d, n, o);
    else k_doubles<<<blocks, 128>>>((const double*)d, n, o);
    const int rc = cudaMemcpy(out, o, (size_t)n * 8, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    cudaFree(o);
    return rc;
}
