// Leaves a pattern in the shared memory of every SM: a CTA that takes a whole SM's worth, several per SM.
#include <cuda_runtime.h>

__global__ void k_fill(unsigned long long word, int words) {
	extern __shared__ unsigned long long s[];
	volatile unsigned long long* v = s;
	for (int k = threadIdx.x; k < words; k += blockDim.x) v[k] = word;
}

extern "C" int fill_shared(unsigned long long word) {
	int device = 0, sms = 0, bytes = 0;
	cudaError_t e = cudaGetDevice(&device);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(k_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
	if (e != cudaSuccess) return (int) e;
	k_fill<<<8 * sms, 256, bytes>>>(word, bytes / 8);
	e = cudaGetLastError();
	if (e == cudaSuccess) e = cudaDeviceSynchronize();
	return (int) e;
}
