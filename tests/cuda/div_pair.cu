// sqrt_recip, recip_rn, div_rn and div_rn2 (tss_device.cuh) against CUDA's IEEE square
// root, reciprocal and division, bit for bit:
//   every x in [2^-100, 2^10]: the square root s and its reciprocal y;
//   every significand b at five exponents: the reciprocal (for the all-ones one the
//     theorem does not promise it);
//   the all-ones divisor under every numerator of two binades;
//   2^33 quotients a / b of seeded significands and exponents, every second one made so
//     that a / b is as near as a float a brings it to a rounding boundary.
// Prints "mismatches <count> of <checked>"; exits 0 unless a CUDA call fails.  The
// kernels touch no memory but one counter.
#include <cstdio>

#include "../../twoscalesplit_gb300/csrc/tss_device.cuh"

using namespace tss;
typedef unsigned long long u64;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ bool recip_ok(float b, float y) { return same(y, __frcp_rn(b)); }

__global__ void k_sqrt(unsigned lo, u64 n, u64* bad) {
    u64 nbad = 0;
    for (u64 t = blockIdx.x * static_cast<u64>(blockDim.x) + threadIdx.x; t < n; t += static_cast<u64>(gridDim.x) * blockDim.x) {
        const float x = __uint_as_float(lo + static_cast<unsigned>(t));
        float y;
        const float s = sqrt_recip(x, y);
        nbad += !(same(s, __fsqrt_rn(x)) && recip_ok(s, y));
    }
    if (nbad) atomicAdd(bad, nbad);
}

__global__ void k_recip(u64* bad) {
    u64 nbad = 0;
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 23); m += stride)
        for (unsigned e = 47; e <= 207; e += 40) {  // 2^-80 ... 2^80
            const float b = __uint_as_float((e << 23) | m);
            nbad += !recip_ok(b, recip_rn(b));
        }
    if (nbad) atomicAdd(bad, nbad);
}

__global__ void k_ones(u64* bad) {
    u64 nbad = 0;
    const float b = __uint_as_float(0x3fffffffu);  // 2 - 2^-23
    const unsigned stride = gridDim.x * blockDim.x;
    for (unsigned m = blockIdx.x * blockDim.x + threadIdx.x; m < (1u << 24); m += stride) {
        const float a = __uint_as_float((126u << 23) + m);  // [0.5, 2)
        const float y = recip_rn(b), ref = __fdiv_rn(a, b);
        const float2 q2 = div_rn2(make_float2(a, -a), b, y);
        nbad += !(same(div_rn(a, b, y), ref) && same(q2.x, ref) && same(q2.y, -ref));
    }
    if (nbad) atomicAdd(bad, nbad);
}

__device__ u64 mix(u64 z) {  // SplitMix64 (G. Steele et al., 2014)
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__global__ void k_div(u64 n, u64* bad) {
    u64 nbad = 0;
    for (u64 t = blockIdx.x * static_cast<u64>(blockDim.x) + threadIdx.x; t < n; t += static_cast<u64>(gridDim.x) * blockDim.x) {
        const u64 z = mix(t), w = mix(z);
        const unsigned eb = 97 + static_cast<unsigned>((z >> 46) % 61), eq = 97 + static_cast<unsigned>((w >> 46) % 61);
        const float b = __uint_as_float((eb << 23) | static_cast<unsigned>(z & 0x7fffffu));
        const float q = __uint_as_float((eq << 23) | static_cast<unsigned>(w & 0x7fffffu));
        float a = q;
        if (t & 1) {  // b times the midpoint above q
            const double mid = 0.5 * (static_cast<double>(q) + static_cast<double>(__uint_as_float(__float_as_uint(q) + 1)));
            a = static_cast<float>(static_cast<double>(b) * mid);
        }
        const float y = recip_rn(b), ref = __fdiv_rn(a, b);
        const float2 q2 = div_rn2(make_float2(a, -a), b, y);
        nbad += !(same(div_rn(a, b, y), ref) && same(q2.x, ref) && same(q2.y, -ref));
    }
    if (nbad) atomicAdd(bad, nbad);
}

int main() {
    u64* d_bad = nullptr;
    int sms = 0;
    if (cudaMalloc(&d_bad, sizeof(u64)) != cudaSuccess) return 1;
    cudaMemset(d_bad, 0, sizeof(u64));
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, 0);
    u64 checked = 0, total = 0;
    const unsigned lo = (127u - 100u) << 23, hi = (127u + 10u) << 23;
    const u64 ndiv = 1ull << 33;
    for (int part = 0; part < 4; ++part) {
        u64 n = 0, nb = 0;
        cudaMemset(d_bad, 0, sizeof(u64));
        if (part == 0) k_sqrt<<<sms * 8, 256>>>(lo, n = static_cast<u64>(hi - lo) + 1, d_bad);
        if (part == 1) k_recip<<<sms * 8, 256>>>(d_bad), n = 5ull << 23;
        if (part == 2) k_ones<<<sms * 8, 256>>>(d_bad), n = 1ull << 24;
        if (part == 3) k_div<<<sms * 8, 256>>>(n = ndiv, d_bad);
        const cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) {
            std::printf("CUDA error: %s\n", cudaGetErrorString(e));
            return 1;
        }
        cudaMemcpy(&nb, d_bad, sizeof(nb), cudaMemcpyDeviceToHost);
        std::printf("part %d: %llu of %llu\n", part, nb, n);
        total += nb;
        checked += n;
    }
    std::printf("mismatches %llu of %llu\n", total, checked);
    cudaFree(d_bad);
    return 0;
}
