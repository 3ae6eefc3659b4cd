// rcp_rn and quot_rn against the division on deterministic pseudo-random
// operands: b of order one (2^-12 .. 2^12), a from 2^-200 to 2^20 and zero, a
// quarter of the significands at the edges (all ones, one bit, their
// neighbours); and infinite numerators.  Prints the differing reciprocals, the differing
// quotients (of 2^28 pairs), the largest relative error of the hardware's
// approximation in units of 2^-19 (rounded up), the differing infinite quotients and
// the square roots (sqrt_nr) that differ.
// Built and run by tests/test_gpu_quotient.py.
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
__device__ double operand(unsigned long long r, int lo, int hi) {
    unsigned long long m = r & 0xfffffffffffffull;
    if ((r >> 62) == 0) {
        const int bit = int((r >> 54) & 0xff) % 52;
        const int kind = int(r >> 52) & 3;
        m = kind == 0 ? (~0ull << bit) : kind == 1 ? (1ull << bit) : kind == 2 ? (1ull << bit) - 1 : ~0ull - (r & 7);
        m &= 0xfffffffffffffull;
    }
    const unsigned long long e = 1023 + lo + (mix64(r + 17) >> 8) % (unsigned)(hi - lo + 1);
    const unsigned long long s = mix64(r + 99) & 0x8000000000000000ull;
    return __longlong_as_double((long long)(s | e << 52 | m));
}
__global__ void k(unsigned long long* bad) {
    const unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long br = 0, bq = 0, err = 0, bi = 0, bs = 0;
    for (int j = 0; j < 64; ++j) {
        const unsigned long long r = mix64(i * 64 + j + 1);
        const double b = operand(mix64(r ^ 0x1234567), -12, 12);
        double a = operand(mix64(r ^ 0xabcdef89), -200, 20);
        if ((r & 0xff) == 0) a = 0.0;
        const double y = rcp_rn(b);
        if (y != 1.0 / b) ++br;
        if (quot_rn(a, b, y) != a / b) ++bq;
        double y0;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
        const unsigned long long e = (unsigned long long)ceil(fabs(fma(-b, y0, 1.0)) * 524288.0);
        err = e > err ? e : err;
        const double inf = __longlong_as_double(0x7ff0000000000000ll);
        if (quot_rn(inf, b, y) != inf / b) ++bi;
        const double x = fabs(a);
        if (sqrt_nr(x) != sqrt(x)) ++bs;
    }
    if (br) atomicAdd(bad, br);
    if (bq) atomicAdd(bad + 1, bq);
    atomicMax(bad + 2, err);
    if (bi) atomicAdd(bad + 3, bi);
    if (bs) atomicAdd(bad + 4, bs);
}
int main() {
    unsigned long long *d, h[5] = {1, 1, 1, 1, 1};
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof(h));
    k<<<(1 << 22) / 256, 256>>>(d);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    printf("err %d reciprocals %llu quotients %llu approx %llu infinite %llu roots %llu\n", int(e), h[0], h[1],
           h[2], h[3], h[4]);
    return e == cudaSuccess ? 0 : 1;
}
