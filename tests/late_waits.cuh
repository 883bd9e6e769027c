// late_waits.cuh - compiled into a build of the library for test_late_waits_gpu.py: now and then a wait for another CTA of the row gives up
// at once, in one thread or in all threads of a CTA, while what it waits for is still on its way.
#pragma once
#ifdef __CUDACC__
static __device__ __forceinline__ int looks_before_giving_up() {
    unsigned long long now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    auto mix = [](unsigned h) {
        h = (h ^ (h >> 16)) * 0x7feb352du;
        h = (h ^ (h >> 15)) * 0x846ca68bu;
        return h ^ (h >> 16);
    };
    const bool full_row = blockDim.x == 512;   // (many more threads wait, and more often)
    const unsigned thread = mix((unsigned)clock64() ^ (threadIdx.x * 2654435761u) ^ (blockIdx.x << 20)), cta = mix((unsigned)(now >> 10) ^ (blockIdx.x << 16));
    if (thread % (full_row ? 100000u : 3000u) == 0u || cta % (full_row ? 400u : 200u) == 0u) return (int)(thread >> 30);
    return 1 << 14;
}
#define FSB_INBOX_LOOKS looks_before_giving_up()
#endif
