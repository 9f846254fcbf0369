// tether_radius (tss_device.cuh) against the FP64 expression it stands for, bit for bit,
// on 2^30 seeded densities and masses: half in the ranges of the workloads, half over
// the floats' whole range (zero, subnormal, infinite and NaN among them).
// Prints "mismatches <count> of <n>"; exits 0 unless a CUDA call fails.  The kernel
// touches no memory but one counter.
#include <cstdio>

#include "../../twoscalesplit_gb300/csrc/tss_device.cuh"

using namespace tss;
typedef unsigned long long u64;

__device__ u64 mix(u64 z) {  // SplitMix64 (G. Steele et al., 2014)
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__global__ void k_check(u64 n, u64* bad) {
    u64 nbad = 0;
    for (u64 t = blockIdx.x * static_cast<u64>(blockDim.x) + threadIdx.x; t < n; t += static_cast<u64>(gridDim.x) * blockDim.x) {
        const u64 z = mix(t);
        const bool wide = t & 1;
        // mass 2^-30 ... 2^3, density 2^-2 ... 2^14
        const float m = __uint_as_float(wide ? static_cast<unsigned>(z >> 33) : ((97u + static_cast<unsigned>(z >> 58) % 33u) << 23) | (static_cast<unsigned>(z >> 32) & 0x7fffffu));
        const float rho = __uint_as_float(wide ? static_cast<unsigned>(z) : ((125u + static_cast<unsigned>(z >> 24) % 16u) << 23) | (static_cast<unsigned>(z) & 0x7fffffu));
        Params P{};
        P.mL = m;
        const double K = 0.5625 * static_cast<double>(m) / kPi;
        P.trK = make_float2(static_cast<float>(K), 0.0f);
        P.trK.y = static_cast<float>(K - static_cast<double>(P.trK.x));
        const float a = tether_radius(P, rho);
        const float b = static_cast<float>(0.75 * sqrt(static_cast<double>(m) / (static_cast<double>(rho) * kPi)));
        nbad += !(__float_as_uint(a) == __float_as_uint(b) || (isnan(a) && isnan(b)));
    }
    if (nbad) atomicAdd(bad, nbad);
}

int main() {
    u64 *d_bad = nullptr, bad = 0;
    const u64 n = 1ull << 30;
    int sms = 0;
    if (cudaMalloc(&d_bad, sizeof(u64)) != cudaSuccess) return 1;
    cudaMemset(d_bad, 0, sizeof(u64));
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
    k_check<<<sms * 8, 256>>>(n, d_bad);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        std::printf("CUDA error: %s\n", cudaGetErrorString(e));
        return 1;
    }
    cudaMemcpy(&bad, d_bad, sizeof(bad), cudaMemcpyDeviceToHost);
    std::printf("mismatches %llu of %llu\n", bad, n);
    cudaFree(d_bad);
    return 0;
}
