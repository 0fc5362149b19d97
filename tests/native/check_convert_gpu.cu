// check_convert_gpu.cu -- on the GPU, for every v in [0, 2^31 - 1]: the words that the
// tensor-core kernels make of v by one fused multiply-add (f64_bits_fma, f32_bits_fma)
// where they do not leave it out, and those of their general path (f64_bits_to_p,
// f32_bits_fp), against v * (1.0 / (2^31 - 1)) by the GPU's own fp64 multiply.
#include <cstdio>

#include "mrg8g_device.cuh"

using namespace mrg8g;

struct Counts {
    unsigned long long seen, fma64, fma32, general64, general32, rare64, rare32;
};

__global__ void k_check(Counts* c) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= kP; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = (uint32_t)i;
        const double u = __dmul_rn((double)v, 1.0 / 2147483647.0);
        const uint64_t want64 = (uint64_t)__double_as_longlong(u);
        const uint32_t want32 = __float_as_uint(__double2float_rn(u));
        uint32_t xn;
        float fh;
        const uint64_t got64 = f64_bits_fma(v, xn);
        const uint32_t got32 = f32_bits_fma(v, fh);
        if (f64_fma_rare(xn)) atomicAdd(&c->rare64, 1ull);
        else if (got64 != want64) atomicAdd(&c->fma64, 1ull);
        if (f32_fma_rare(fabsf(__fsub_rn(fh, 0.5f)))) atomicAdd(&c->rare32, 1ull);
        else if (got32 != want32) atomicAdd(&c->fma32, 1ull);
        if (f64_bits_to_p(v) != want64) atomicAdd(&c->general64, 1ull);
        if (f32_bits_fp(v) != want32) atomicAdd(&c->general32, 1ull);
    }
    if (threadIdx.x == 0) atomicAdd(&c->seen, 1ull);
}

int main() {
    Counts* d = nullptr;
    Counts c{};
    if (cudaMalloc(&d, sizeof(c)) || cudaMemset(d, 0, sizeof(c))) return 2;
    k_check<<<1024, 256>>>(d);
    if (cudaGetLastError() || cudaMemcpy(&c, d, sizeof(c), cudaMemcpyDeviceToHost)) return 2;
    std::printf("blocks %llu, wrong: fma %llu %llu, general %llu %llu; left out %llu %llu\n", c.seen, c.fma64, c.fma32,
                c.general64, c.general32, c.rare64, c.rare32);
    return c.seen != 1024 || c.fma64 || c.fma32 || c.general64 || c.general32 || !c.rare64 || c.rare64 > 1024 ||
           !c.rare32 || c.rare32 > 4096;
}
