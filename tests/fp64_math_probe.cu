// Element-wise access to the primitives of sph_math.cuh, and the FP32 quotient of the ghost stencils, for test_fp64_math_gpu.py.
#include "sph_math.cuh"

using namespace sph;

__global__ void k_probe(int op, long long n, const double* a, const double* b, double* out, const double* tab, int p, int q, double c) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = a[i], y = b[i];
    switch (op) {
        case 0: out[i] = near_div(x, y); break;
        case 2: out[i] = fast_sqrt(x); break;
        case 3: out[i] = fast_pow(tab, x, c); break;
        case 5: out[i] = gdiv((float)x, (float)y); break;
        default: {
            const double e = (double)p / q;
            out[i] = root_pow(x, p, q, (q + 1.0) / (q - 1.0), (float)e, (float)(e - (double)(float)e));
        }
    }
}

extern "C" int probe(int op, long long n, const double* a, const double* b, double* out, int p, int q, double c) {
    double h[kPowTab], *da = nullptr, *db = nullptr, *dout = nullptr, *tab = nullptr;
    fill_pow_tables(h);
    const size_t bytes = sizeof(double) * (size_t)n;
    cudaError_t e = cudaMalloc((void**)&da, bytes);
    if (e == cudaSuccess) e = cudaMalloc((void**)&db, bytes);
    if (e == cudaSuccess) e = cudaMalloc((void**)&dout, bytes);
    if (e == cudaSuccess) e = cudaMalloc((void**)&tab, sizeof(h));
    if (e == cudaSuccess) e = cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(tab, h, sizeof(h), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_probe<<<(unsigned)((n + 255) / 256), 256>>>(op, n, da, db, dout, tab, p, q, c);
        e = cudaMemcpy(out, dout, bytes, cudaMemcpyDeviceToHost);
    }
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    cudaFree(tab);
    return (int)e;
}
