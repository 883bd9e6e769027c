// full_row_math.cu - the exponential and the division of the full-vocabulary kernel over arrays, for the tests: the kernel's
// own source is compiled in, so that what is tested is what it runs.
#include "../ferro_b200/csrc/fsb_fullrow.cu"

namespace fsb {
namespace {
// diff[i] <= 0 and temp[i] > 0: quotient (x - max) / T as the kernel forms it and as the device divides, and the weight
// exp((x - max) / T) in units of 2^-62 (no logit lies below the cut: diff >= -45 temp).
__global__ void math_kernel(const float* diff, const float* temp, int n, double* quotient, double* divided, u64* weight) {
    __shared__ double table[64];
    if (threadIdx.x < 64) table[threadIdx.x] = exp2((double)threadIdx.x / 64.0);
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        RowCtx rc{};
        rc.mx = 0.0f;
        rc.temp = (double)temp[i];
        rc.inv_temp = __ddiv_rn(1.0, rc.temp);
        rc.cut = -45.0f * temp[i];
        rc.table = table;
        quotient[i] = rc.scaled(diff[i]);
        divided[i] = __ddiv_rn((double)diff[i], rc.temp);
        weight[i] = rc.weight(diff[i]).value();
    }
}
}  // namespace
}  // namespace fsb

extern "C" __attribute__((visibility("default"))) int full_row_math(const float* diff, const float* temp, int n, double* quotient, double* divided,
                                                                   unsigned long long* weight) {
    fsb::math_kernel<<<296, 256>>>(diff, temp, n, quotient, divided, weight);
    if (cudaGetLastError() != cudaSuccess) return 1;
    return (int)cudaDeviceSynchronize();
}
