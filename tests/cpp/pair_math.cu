// Device functions of the pair kernels (sf_pairs.cuh) over arrays, for
// tests/test_gpu_pair_math.py.  run() returns a CUDA error code.
#include "sf_pairs.cuh"

using namespace n2p2b200;

static __global__ void kMath(int n, const double* s, const double* c, const double* tab, double* expD, double* wideD,
                      double* rootD, float* expF, float* rootF)
{
    __shared__ double t[64];
    if (threadIdx.x < 64) t[threadIdx.x] = tab[threadIdx.x];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    expD[i] = expScaled<false>(s[i], c[i], t);
    wideD[i] = expScaled<true>(s[i], c[i], t);
    rootD[i] = invSqrt(s[i]);
    expF[i] = expScaled<false>((float)s[i], (float)c[i], t);   // FP32: c of 2^(c s)
    rootF[i] = invSqrt((float)s[i]);
}

extern "C" int run(int n, const double* s, const double* c, const double* tab, double* expD, double* wideD,
                   double* rootD, float* expF, float* rootF)
{
    double* d = nullptr;
    cudaError_t e = cudaMalloc((void**)&d, sizeof(double) * (6 * (size_t)n + 64));
    if (e != cudaSuccess) return (int)e;
    double *ds = d, *dc = d + n, *dt = d + 2 * n, *oe = d + 2 * n + 64, *ow = oe + n, *orr = ow + n;
    float *fe = reinterpret_cast<float*>(orr + n), *fr = fe + n;
    cudaMemcpy(ds, s, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(dc, c, sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(dt, tab, sizeof(double) * 64, cudaMemcpyHostToDevice);
    kMath<<<(n + 127) / 128, 128>>>(n, ds, dc, dt, oe, ow, orr, fe, fr);
    cudaMemcpy(expD, oe, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(wideD, ow, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(rootD, orr, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(expF, fe, sizeof(float) * n, cudaMemcpyDeviceToHost);
    e = cudaMemcpy(rootF, fr, sizeof(float) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
