// fp64_ops.cu -- the branch-free division and square root of flux_fp64.cuh
// on arrays and on random operands, for test_gpu_fp64_ops.py. Compiled by
// that test with the plain FP64 form's flags.
#include <cstdint>

#include "device_common.cuh"
#include "flux_fp64.cuh"

using namespace amrgpu;

namespace {

__device__ double apply(int op, double a, double b)
{
    if (op == 0) return recip_rn(b);
    if (op == 1) return sqrt_rn(b);
    return quotient_by(a, b, recip_rn(b));
}

__device__ double ieee(int op, double a, double b)
{
    if (op == 0) return 1.0 / b;
    if (op == 1) return sqrt(b);
    return a / b;
}

__device__ uint64_t mix(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// mantissa by turns random, near the binade's upper and lower end; exponent
// in [lo, hi]
__device__ double operand(uint64_t r, int turn, int lo, int hi)
{
    const uint64_t s = mix(r ^ 0x5bd1e995u);
    uint64_t m = r;
    if (turn == 1) m = ~(r & 1023);
    if (turn == 2) m = r & 1023;
    const int e = lo + (int)(s % (uint64_t)(hi - lo + 1));
    return __longlong_as_double((long long)((m & 0xfffffffffffffull) | ((uint64_t)(1023 + e) << 52)));
}

__global__ void array_kernel(int op, const double *a, const double *b, double *out, long long n)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
        out[k] = apply(op, a[k], b[k]);
}

// a: numerators with exponents in [alo, ahi]; one turn in four is b times a
// mantissa, moved by at most a place: a quotient next to a double
__global__ void random_kernel(int op, uint64_t seed, long long n, int alo, int ahi, int blo, int bhi,
                              unsigned long long *bad)
{
    unsigned long long mine = 0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        const uint64_t r1 = mix(seed + (uint64_t)k), r2 = mix(r1 + 77), r3 = mix(r2 + 5);
        const double b = operand(r1, (int)(k & 3), blo, bhi);
        double a = operand(r2, (int)(k >> 2 & 3), alo, ahi);
        if (op == 2 && (k >> 4 & 3) == 3)
            a = __longlong_as_double(__double_as_longlong(b * operand(r2, 0, 0, 0)) + (long long)(r3 % 3) - 1);
        if (r3 & (1ull << 60)) a = -a;
        if (__double_as_longlong(apply(op, a, b)) != __double_as_longlong(ieee(op, a, b))) ++mine;
    }
    if (mine) atomicAdd(bad, mine);
}

}  // namespace

// op: 0 1/b, 1 sqrt(b), 2 a/b. 0 or a CUDA error.
extern "C" int fp64_ops(int op, const double *a, const double *b, double *out, long long n)
{
    double *d = nullptr;
    const size_t bytes = sizeof(double) * (size_t)n;
    cudaError_t e = cudaMalloc(&d, 3 * bytes);
    if (e != cudaSuccess) return (int)e;
    if (e == cudaSuccess) e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        array_kernel<<<148 * 4, 256>>>(op, d, d + n, d + 2 * n, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}

// *bad: how many of n random operands differ from the IEEE operation in any
// bit. 0 or a CUDA error.
extern "C" int fp64_random(int op, unsigned long long seed, long long n, int alo, int ahi, int blo, int bhi,
                           unsigned long long *bad)
{
    unsigned long long *d = nullptr;
    cudaError_t e = cudaMalloc(&d, sizeof(*d));
    if (e != cudaSuccess) return (int)e;
    e = cudaMemset(d, 0, sizeof(*d));
    if (e == cudaSuccess) {
        random_kernel<<<148 * 8, 256>>>(op, seed, n, alo, ahi, blo, bhi, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(bad, d, sizeof(*d), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}

namespace {

__global__ void marked_kernel(const double *q, int *marked, int n)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double P[9];
    cell_prims_fp64(q + 4 * k, P);
    marked[k] = __double2hiint(P[8]) < 0;
}

}  // namespace

// Whether the records of n states [n][4] are marked. 0 or a CUDA error.
extern "C" int fp64_marked(const double *q, int *marked, int n)
{
    double *d = nullptr;
    const size_t in = sizeof(double) * 4 * (size_t)n, out = sizeof(int) * (size_t)n;
    cudaError_t e = cudaMalloc(&d, in + out);
    if (e != cudaSuccess) return (int)e;
    int *m = reinterpret_cast<int *>(d + 4 * (size_t)n);
    e = cudaMemcpy(d, q, in, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        marked_kernel<<<(n + 255) / 256, 256>>>(d, m, n);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(marked, m, out, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
