// Every float through the colour transfer's table encode and through the exact
// encode it stands for (image360_b200/csrc/color.cu, compiled here with the
// library's flags): prints the number of floats whose codes differ, the number
// of steps that the exact encode takes elsewhere than the table says, and the
// number of floats at which it falls.  Exit code 0: all are 0.
#include "../image360_b200/csrc/color.cu"

#include <cstdio>

namespace i360b
{
int device() { return 0; }
int sm_count() { return 148; }
int fail(int code, const char*, ...) { return code; }
int cuda_fail(cudaError_t, const char*) { return I360B_CUDA_ERROR; }
int check_launch(const char*) { return cudaGetLastError() == cudaSuccess ? I360B_SUCCESS : I360B_CUDA_ERROR; }
int dev_alloc(void** p, size_t bytes, cudaStream_t s, const char*)
{
    return cudaMallocAsync(p, bytes, s) == cudaSuccess ? I360B_SUCCESS : I360B_CUDA_ERROR;
}
void dev_free(void* p, cudaStream_t s) { cudaFreeAsync(p, s); }
}  // namespace i360b

__global__ void k_every_float(unsigned long long* differ, unsigned long long* falls)
{
    const unsigned long long n = 1ull << 32;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x)
    {
        const float c = __uint_as_float((uint32_t)i);
        const unsigned exact = encode_u16(c < 0.0f ? 0.0f : c);  // (as lab_to_rgb)
        if (encode_u16_table(c) != exact) atomicAdd(differ, 1ull);
        if (i > 0 && i <= 0x7f800000u && encode_u16(__uint_as_float((uint32_t)i - 1)) > exact) atomicAdd(falls, 1ull);
    }
}

__global__ void k_every_step(unsigned long long* wrong)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 65535) return;
    const float s = g_encodeStep[k];
    if (!(encode_u16(s) > k && encode_u16(__uint_as_float(__float_as_uint(s) - 1)) <= k)) atomicAdd(wrong, 1ull);
}

int main()
{
    unsigned long long *d, h[3] = {~0ull, ~0ull, ~0ull};
    if (ensure_tables(nullptr) != I360B_SUCCESS || cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 2;
    cudaMemset(d, 0, sizeof(h));
    k_every_step<<<256, 256>>>(d);
    k_every_float<<<148 * 8, 256>>>(d + 1, d + 2);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("steps elsewhere %llu, floats that differ %llu, floats at which the encode falls %llu\n", h[0], h[1], h[2]);
    return h[0] || h[1] || h[2] ? 1 : 0;
}
