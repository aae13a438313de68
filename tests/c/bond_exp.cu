/*
 * Exhaustive comparison of the Wolff bond test (xy_device.cuh) with its
 * definition, active iff J r_i r_j > 0 and u < 1 - exp(-2 beta J r_i r_j) with
 * CUDA's __expf and u = (word >> 8) 2^-24: every FP32 product J r_i r_j, each with
 * the words on both sides of the threshold and at the ends of the range; the
 * scalar form and the packed one.  Prints the number of differences.
 */
#include <cstdint>
#include <cstdio>

#include "xy_device.cuh"

__global__ void compare(unsigned long long* bad) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long n = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < 1ull << 32; i += step) {
        const float prod = __uint_as_float((uint32_t)i);
        const float p = __fsub_rn(1.0f, __expf(__fmul_rn(-1.0f, prod)));
        const bool positive = prod > 0.0f;
        const uint32_t k = positive ? (uint32_t)__fmul_rn(p, 16777216.0f) : 0u; /* p is a multiple of 2^-24, at most 1 */
        const uint32_t words[6] = {k << 8, (k << 8) - 1u, (k << 8) + 1u, ((k + 1u) << 8) - 1u, 0u, 0xffffffffu};
        for (int w = 0; w < 6; ++w) {
            const bool want = positive && slsf_u24f(words[w]) < p;
            n += slsf::wolff_bond_active(1.0f, prod, 1.0f, -1.0f, words[w]) != want;
            uint32_t a, b;
            slsf::wolff_bond_words(make_float2(prod, prod), make_float2(-1.0f, -1.0f), words[w], words[5 - w], a, b);
            n += (a >> lane & 1u) != (uint32_t)want;
            n += (b >> lane & 1u) != (uint32_t)(positive && slsf_u24f(words[5 - w]) < p);
        }
    }
    atomicAdd(bad, n);
}

int main() {
    unsigned long long *bad = nullptr, host = ~0ull;
    if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess || cudaMemset(bad, 0, sizeof(*bad)) != cudaSuccess) return 3;
    compare<<<4096, 256>>>(bad);
    if (cudaGetLastError() != cudaSuccess || cudaMemcpy(&host, bad, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    std::printf("differences %llu\n", host);
    cudaFree(bad);
    return host ? 1 : 0;
}
