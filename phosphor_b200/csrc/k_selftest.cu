// k_selftest.cu — the kernels' short forms of quotients and exponentials, element by element, for
// the tests that compare them with the operations they stand for.
#include "dev_shading.cuh"
#include "gather_walk.cuh"
#include "kernels.hpp"

namespace phx {

__global__ void k_selftest_math(int fn, const float *a, const float *b, float *out, u32 n) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const float x = a[i], y = b[i];
    float r = 0.0f;
    switch (fn) {
    case 0: r = unorm8((u8)x); break;
    case 1: r = div_zero(x, y); break;
    case 2: r = div_known(x, y, 1.0f / y); break;
    case 3: r = div_gauss(x); break;
    case 4: r = exp_unit(x); break;
    case 5: r = pm_expf(x); break;
    }
    out[i] = r;
}

cudaError_t selftest_math(int fn, const float *a, const float *b, float *out, u32 n) {
    const size_t bytes = 4 * (size_t)n;
    float *d = nullptr;
    cudaError_t e = cudaMalloc((void **)&d, 3 * bytes);
    if (e != cudaSuccess)
        return e;
    float *da = d, *db = d + n, *dout = d + 2 * (size_t)n;
    if ((e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice)) == cudaSuccess &&
        (e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice)) == cudaSuccess) {
        k_selftest_math<<<(n + 255) / 256, 256>>>(fn, da, db, dout, n);
        if ((e = cudaGetLastError()) == cudaSuccess)
            e = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    }
    cudaFree(d);
    return e;
}

} // namespace phx
