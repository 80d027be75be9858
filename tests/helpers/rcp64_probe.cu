// The pair kernels' FP64 reciprocal over an array.
#include "pair_common.cuh"

__global__ void k_rcp64(const double* x, double* y, int n) {
	const int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) y[i] = mdgpu::rcp64(x[i]);
}

extern "C" int rcp64_of(const double* x, double* y, int n) {
	double *dx = nullptr, *dy = nullptr;
	cudaError_t e = cudaMalloc(&dx, sizeof(double) * n);
	if (e == cudaSuccess) e = cudaMalloc(&dy, sizeof(double) * n);
	if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice);
	if (e == cudaSuccess) {
		k_rcp64<<<(n + 255) / 256, 256>>>(dx, dy, n);
		e = cudaMemcpy(y, dy, sizeof(double) * n, cudaMemcpyDeviceToHost);
	}
	cudaFree(dx);
	cudaFree(dy);
	return (int) e;
}
