// The kernels' divisions and reciprocal (models.cuh, tc_common.cuh) beside the operator, on
// random normal numbers: for each the largest difference in units of the last place and how
// many quotients differ, written to out[2 * form + {0, 1}].
#include "../cubnm_b200/csrc/models.cuh"
#include "../cubnm_b200/csrc/tc_common.cuh"

namespace {

__device__ unsigned long long mix(unsigned long long x) {   // splitmix64
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
// +-[1, 2) 2^e, e in [-range, range)
__device__ double number(unsigned long long i, int range) {
    const unsigned long long h = mix(i);
    const double m = 1.0 + (double)(h >> 12) * 0x1p-52;
    return scalbn(h & 1 ? -m : m, (int)((h >> 1) % (2 * range)) - range);
}
__device__ void note(unsigned long long *out, int form, unsigned long long ulps) {
    atomicMax(out + 2 * form, ulps);
    if (ulps) atomicAdd(out + 2 * form + 1, 1ull);
}

__global__ void k_check(unsigned long long *out, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double a = number(3ull * i, 200), b = number(3ull * i + 1, 200);
        const float af = (float)number(3ull * i, 40), bf = (float)number(3ull * i + 1, 40);
        note(out, 0, llabs(__float_as_int(cbnm::div_nr(af, bf)) - (long long)__float_as_int(af / bf)));
        note(out, 1, llabs(__double_as_longlong(cbnm::div_nr(a, b)) - __double_as_longlong(a / b)));
        note(out, 2, llabs(__double_as_longlong(cbnm::rcp_fast(b)) - __double_as_longlong(1.0 / b)));
    }
}

}  // namespace

extern "C" int division_check(unsigned long long *host, int n) {
    unsigned long long *out;
    if (cudaMalloc(&out, 6 * sizeof(*out)) != cudaSuccess) return 1;
    cudaMemset(out, 0, 6 * sizeof(*out));
    k_check<<<592, 256>>>(out, n);
    const cudaError_t e = cudaMemcpy(host, out, 6 * sizeof(*out), cudaMemcpyDeviceToHost);
    cudaFree(out);
    return e == cudaSuccess ? 0 : 1;
}
