// sqrt_nr against sqrt(): the ends of the exponent range, zeros, infinity, NaN and
// negative numbers bit for bit (every NaN alike); every power of two; 2^24
// pseudo-random numbers of the whole range; and the numbers next to the squares
// of 2^22 midpoints of two neighbouring roots, where a last bit may differ.  Prints
// the special values that differ, the random ones, those next to midpoints, and the
// largest difference in ulps.  Built and run by tests/test_gpu_square_root.py.
#include <cstdio>
#include "lattice.cuh"
using namespace cav;
__device__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    return x ^ (x >> 33);
}
__device__ unsigned long long ulps(double x) {
    const double g = sqrt_nr(x), w = sqrt(x);
    if (isnan(g) && isnan(w)) return 0;
    const long long a = __double_as_longlong(g), b = __double_as_longlong(w);
    return a == b ? 0 : isnan(g) || isnan(w) ? ~0ull : (unsigned long long)(a > b ? a - b : b - a);
}
__global__ void k(const double* special, int n_special, unsigned long long* out) {
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long d, worst = 0;
    if (i < n_special) {
        d = ulps(special[i]);
        if (d) atomicAdd(out, 1ull);
    }
    if (i < 2046) {
        d = ulps(__longlong_as_double((long long)(i + 1) << 52));
        if (d) atomicAdd(out, 1ull);
    }
    for (int j = 0; j < 16; ++j) {
        const unsigned long long r = mix64(i * 16 + j + 1);
        d = ulps(__longlong_as_double((long long)(r & 0x7fffffffffffffffull) % 0x7ff0000000000000ll));
        if (d) atomicAdd(out + 1, 1ull);
        worst = d > worst ? d : worst;
    }
    for (int j = 0; j < 4; ++j) {
        // (2 m + 1)^2 of 54 bits in two binades, cut to 53 bits, and its neighbours
        const unsigned long long m = mix64(~(i * 4 + j)) & 0xfffffffffffffull;
        const unsigned long long s = (1ull << 53) + 2 * m + 1;  // midpoint, 54 bits
        const unsigned __int128 sq = (unsigned __int128)s * s;
        const int sh = (sq >> 107) ? 55 : 54;
        const long long c = (long long)(sq >> sh);
        for (int o = -1; o <= 2; ++o) {
            // the parity of the exponent that makes sqrt's significand s
            const double x = ldexp(double(c + o), sh - 106);
            d = ulps(x);
            if (d) atomicAdd(out + 2, 1ull);
            worst = d > worst ? d : worst;
        }
    }
    atomicMax(out + 3, worst);
}
int main() {
    const double inf = INFINITY;
    const double sp[] = {0.0, -0.0, inf, -inf, NAN, -1.0, -0x1p-1074, 0x1p-1074, 0x1p-1073, 0x1.8p-1073, 0x1p-1022,
                         0x1.fffffffffffffp-1023, 0x1.fffffffffffffp-701, 0x1p-700, 0x1.fffffffffffffp-961, 0x1p-960,
                         0x1.fffffffffffffp700, 0x1p701, 0x1.fffffffffffffp960, 0x1.0000000000001p960, 0x1p1023,
                         0x1.fffffffffffffp1023, 1e-300, 1e300};
    constexpr int n = sizeof(sp) / sizeof(sp[0]);
    double* ds;
    unsigned long long *d, h[4] = {1, 1, 1, 1};
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMalloc(&ds, sizeof(sp)) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof(h));
    cudaMemcpy(ds, sp, sizeof(sp), cudaMemcpyHostToDevice);
    k<<<(1 << 20) / 256, 256>>>(ds, n, d);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    printf("err %d special %llu random %llu midpoint %llu worst %llu\n", int(e), h[0], h[1], h[2], h[3]);
    return e == cudaSuccess ? 0 : 1;
}
