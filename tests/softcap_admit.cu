// softcap_admit.cu - the streaming kernel's early bound under the softcap over arrays, for the tests: the kernel's own source is compiled in.
#include "../ferro_b200/csrc/fsb_device.cuh"

namespace fsb {
namespace {
__global__ void admit_kernel(const float* thr, const float* cap, int n, float* admit) {   // a warp per pair
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        float a = -FLT_MAX, seen = 0.0f;
        softcap_admit(thr[i], cap[i], a, seen);
        if (threadIdx.x == 0) admit[i] = a;
    }
}
}  // namespace
}  // namespace fsb

extern "C" __attribute__((visibility("default"))) int softcap_admit_of(const float* thr, const float* cap, int n, float* admit) {
    fsb::admit_kernel<<<296, 32>>>(thr, cap, n, admit);
    if (cudaGetLastError() != cudaSuccess) return 1;
    return (int)cudaDeviceSynchronize();
}
