// tmem_neighbour.cu -- kernels of another library beside the generator's on one
// stream.
//   k_behind  may start while the kernel before it still runs, takes tensor memory
//             first, and only then waits for that kernel and reads its outputs.
//   k_ahead   lets the kernel behind it start at once and takes its own tensor
//             memory some microseconds later.
#include <cuda_runtime.h>
#include <stdint.h>

constexpr uint32_t kCols = 128;

__device__ __forceinline__ void take(uint32_t* tmem) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(tmem)),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void give_back(const uint32_t* tmem) {
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem), "r"(kCols));
}

__global__ void __launch_bounds__(32) k_behind(const uint64_t* in, uint64_t* seen, uint32_t count) {
    __shared__ uint32_t tmem;
    take(&tmem);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (uint32_t i = blockIdx.x * 32 + threadIdx.x; i < count; i += gridDim.x * 32) seen[i] = in[i];
    give_back(&tmem);
}

// At most `us` microseconds (or 2^20 looks at the clock) before it takes its columns.
__global__ void __launch_bounds__(32) k_ahead(uint32_t us, uint32_t* done) {
    __shared__ uint32_t tmem;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    unsigned long long t0, t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    for (int i = 0; i < 1 << 20; ++i) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t - t0 >= us * 1000ull) break;
    }
    __syncwarp();
    take(&tmem);
    if (threadIdx.x == 0) atomicAdd(done, 1u);
    give_back(&tmem);
}

extern "C" int ahead(uint32_t us, void* done, int blocks, void* stream) {
    k_ahead<<<blocks, 32, 0, (cudaStream_t)stream>>>(us, (uint32_t*)done);
    return (int)cudaGetLastError();
}

extern "C" int behind(const void* in, void* seen, uint32_t count, int blocks, void* stream) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)blocks);
    c.blockDim = dim3(32);
    c.stream = (cudaStream_t)stream;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return (int)cudaLaunchKernelEx(&c, k_behind, (const uint64_t*)in, (uint64_t*)seen, count);
}
