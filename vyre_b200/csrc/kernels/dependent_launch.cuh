// Programmatic dependent launch: a kernel that lets_next_start() is joined on the SMs by the next launch of its stream as soon as all
// of its blocks have started, and that launch has its own start (1 to 3 us of launch latency, barriers, tensor memory, descriptors)
// behind it when it comes to waits_for_previous(), which returns when everything before it in the stream is complete and visible.
// Both are no-ops in a plain launch. A kernel that is launched this way calls waits_for_previous() in every thread that reads or
// writes global memory, before it does, since the launch before it may still be waiting for the one before that. What earlier launches may
// still be writing when it starts is no read-only data: neither `__restrict__` nor `__ldg` on its operands, whose loads the compiler may
// move up past the wait, or the hardware serve from lines that nobody invalidates.
// Where a kernel calls lets_next_start(): at its start if what follows does little before its wait; behind its own loads if it is short
// and a projection's prefetch of weights may follow (RMSNorm at 8 rows in front of a projection: 10 us a decode block lost otherwise).
// A kernel with tensor memory calls it when the block has allocated its share: a block of the next launch beside it may take what is left, keeps
// it while it waits for this launch, and an allocation waits without a limit.
// Measured, us a call in chains of submissions, plain / dependent: int4 linear at 48 rows 20.6 / 18.6, published affine-grouped row
// 16.0 / 14.5, affine-grouped decode 36.0 / 35.3, Q4_K linear 24.8 / 23.8; a MoE layer of 64 tokens (six launches) 268 / 257.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace vybk {

__device__ __forceinline__ void lets_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void waits_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependent_start() {
    waits_for_previous();
    lets_next_start();
}
// The line of an address into L2, whose contents stay coherent with what earlier launches still write: allowed before the wait
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

inline void dependent(cudaLaunchAttribute& a) {
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
}
// A caller that leaves SMs free for another kernel does not want the next launch on them early: such a launch neither starts early nor lets the
// next one start (small operators behind a projection would fill the free SM and sit there until it ends), except in chains of constant
// weights, whose launches are meant to overlap.
inline bool whole_device(int dev, int sm_count) {
    int sms = 0;
    return cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sm_count >= sms;
}
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    dependent(attr);
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
// A kernel without shared memory to speak of that runs between kernels that ask for all of it. Left to itself it may be given another
// split between L1 and shared memory, and an SM changes its split only when it is empty: the early start is lost, on some graphs and
// not on others (a decode block at 8 rows 65 or 52 us, from one capture to the next).
template <auto Kernel, typename... A>
cudaError_t launch_between(dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute((const void*)Kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    return launch_dependent(Kernel, grid, block, smem, s, args...);
}

}  // namespace vybk
