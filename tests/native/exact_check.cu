// Comparisons of csrc/sx_exact.cuh with the compiler's correctly rounded operations;
// each kernel adds the number of differences to *bad and of comparisons to *done.
#include <cuda_runtime.h>

#include "sx_exact.cuh"

using u64 = unsigned long long;

__device__ void add(u64* bad, u64* done, u64 b, u64 d) {
    if (b) atomicAdd(bad, b);
    atomicAdd(done, d);
}
// every float with bits in [first, last), both signs
__global__ void rcp_kernel(unsigned first, unsigned last, u64* bad, u64* done) {
    u64 b = 0, d = 0;
    for (u64 i = first + (u64)blockIdx.x * blockDim.x + threadIdx.x; i < last; i += (u64)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)i);
        b += __float_as_uint(sx::rcp_rn(x)) != __float_as_uint(1.0f / x);
        b += __float_as_uint(sx::rcp_rn(-x)) != __float_as_uint(1.0f / -x);
        d += 2;
    }
    add(bad, done, b, d);
}
__global__ void sqrt_kernel(unsigned first, unsigned last, u64* bad, u64* done) {
    u64 b = 0, d = 0;
    for (u64 i = first + (u64)blockIdx.x * blockDim.x + threadIdx.x; i < last; i += (u64)gridDim.x * blockDim.x) {
        const float x = __uint_as_float((unsigned)i);
        b += __float_as_uint(sx::sqrt_rn(x)) != __float_as_uint(sqrtf(x));
        ++d;
    }
    add(bad, done, b, d);
}
// Every pair of significands a, b (24-bit integers) whose quotient lies within reach /
// (b 2^k) of a midpoint m / 2^k of two floats, m odd, 2^24 < m < 2^25: k = 24 for a >= b,
// 25 for a < b.  With rho = a 2^k - b m and b = 2^j c, c odd: rho = 2^j r, r odd, and m = -r
// / c modulo 2^(k-j).  ea, eb: exponents added to a's and b's.
__global__ void div_kernel(int reach, int ea, int eb, u64* bad, u64* done) {
    u64 n = 0, d = 0;
    for (unsigned b = (1u << 23) + blockIdx.x * blockDim.x + threadIdx.x; b < 1u << 24; b += gridDim.x * blockDim.x) {
        const int j = __ffs(b) - 1;
        const unsigned c = b >> j;
        unsigned inv = c;  // 1 / c modulo 2^32: Newton doubles the bits, 3 at first
        for (int i = 0; i < 4; ++i) inv *= 2u - c * inv;
        const float fb = __uint_as_float((unsigned)(127 + eb) << 23 | (b & 0x7fffffu));
        const float y = sx::rcp_rn(fb);
        for (int k = 24; k <= 25; ++k)
            for (int r = 1; (long long)r << j <= reach; r += 2)
                for (int sign = -1; sign <= 1; sign += 2) {
                    const long long rho = (long long)(sign * r) << j;
                    const unsigned mod = 1u << (k - j), m0 = (0u - (unsigned)(sign * r) * inv) & (mod - 1u);
                    for (u64 m = (1u << 24) + ((m0 - (1u << 24)) & (mod - 1u)); m < 1u << 25; m += mod) {
                        const long long num = (long long)b * (long long)m + rho;
                        const unsigned a = (unsigned)(num >> k);
                        if ((long long)a << k != num || a < 1u << 23 || a >= 1u << 24 || (a >= b) != (k == 24)) continue;
                        const float fa = __uint_as_float((unsigned)(127 + ea) << 23 | (a & 0x7fffffu));
                        n += __float_as_uint(sx::div_rn(fa, fb, y)) != __float_as_uint(fa / fb);
                        n += __float_as_uint(sx::div_rn(-fa, fb, y)) != __float_as_uint(-fa / fb);
                        d += 2;
                    }
                }
    }
    add(bad, done, n, d);
}

extern "C" int check(int what, unsigned first, unsigned last, int reach, int ea, int eb, u64* out) {
    u64* dev = nullptr;
    if (cudaMalloc(&dev, 16) != cudaSuccess || cudaMemset(dev, 0, 16) != cudaSuccess) return 1;
    if (what == 0) rcp_kernel<<<1216, 256>>>(first, last, dev, dev + 1);
    if (what == 1) sqrt_kernel<<<1216, 256>>>(first, last, dev, dev + 1);
    if (what == 2) div_kernel<<<1216, 256>>>(reach, ea, eb, dev, dev + 1);
    const bool ok = cudaMemcpy(out, dev, 16, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(dev);
    return ok ? 0 : 2;
}
