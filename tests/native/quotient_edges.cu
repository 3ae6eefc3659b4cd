// rcp_rn and quot_rn against the division, bit for bit (every NaN alike), on
// every pair of the operands where a branch-free form can go wrong: signed
// zeros, infinities, NaN, all-ones significands, very small and very large
// denominators.  Prints the pairs that differ.
// Built and run by tests/test_gpu_quotient_edges.py.
#include <cstdio>
#include <cstring>
#include <cmath>
#include "lattice.cuh"
using namespace cav;
constexpr int NB = 22, NA = 16;
__global__ void k(const double* a, const double* b, double* got, double* want) {
    const int i = threadIdx.x, j = blockIdx.x;
    if (i > NA || j >= NB) return;
    const double y = rcp_rn(b[j]);
    // row NA: the reciprocals
    got[j * (NA + 1) + i] = i == NA ? y : quot_rn(a[i], b[j], y);
    want[j * (NA + 1) + i] = i == NA ? 1.0 / b[j] : a[i] / b[j];
}
int main() {
    const double inf = INFINITY, ones = 1.0 - 0x1p-53;
    const double b[NB] = {0.0,  -0.0, inf,   -inf,   NAN,    1.0,   -1.0,   0.9,   ones,   -ones,  ones / 2,
                          3.0,  -0.7, 1e-12, -1e-12, 1e-300, 1e300, -1e300, 1e100, 0x1p-60, 2.0 / 3.0, 1.5};
    const double a[NA] = {0.0, -0.0, inf, -inf, NAN, 1.0, -1.0, 0.1875, 1e-5, -2.5e-3, 1e-200, -1e-200, ones, 7.0, -0x1p-40, 1e-7};
    double *d, got[NB * (NA + 1)], want[NB * (NA + 1)];
    if (cudaMalloc(&d, sizeof(a) + sizeof(b) + 2 * sizeof(got)) != cudaSuccess) return 1;
    double *da = d, *db = da + NA, *dg = db + NB, *dw = dg + NB * (NA + 1);
    cudaMemcpy(da, a, sizeof(a), cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, sizeof(b), cudaMemcpyHostToDevice);
    k<<<NB, 32>>>(da, db, dg, dw);
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(got, dg, sizeof(got), cudaMemcpyDeviceToHost);
    cudaMemcpy(want, dw, sizeof(want), cudaMemcpyDeviceToHost);
    int bad = 0;
    for (int j = 0; j < NB; ++j)
        for (int i = 0; i <= NA; ++i) {
            const double g = got[j * (NA + 1) + i], w = want[j * (NA + 1) + i];
            if (!std::memcmp(&g, &w, 8) || (std::isnan(g) && std::isnan(w))) continue;
            std::printf("%a / %a: %a, not %a\n", i == NA ? 1.0 : a[i], b[j], g, w);
            ++bad;
        }
    std::printf("err %d differing %d\n", int(e), bad);
    return e == cudaSuccess ? 0 : 1;
}
