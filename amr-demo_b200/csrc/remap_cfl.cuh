// remap_cfl.cuh -- the state remap of an in-place regrid fused with the
// CFL minimum of the remapped state (the next segment's first dt), in one
// pass over the new mesh's cells instead of two.
//
// The remap is remap_kernel's (kernels_misc.cu): refine injects the parent
// patch into each child (solver_refine_operator_2d.F90:49-52), coarsen
// writes (uc1+uc2+uc3+uc4)*0.25 (solver_coarsen_operator_2d.F90:49-50).
// Each cell's CFL candidate is then taken from the values just written, by
// the candidate functor of the form's CFL prologue kernel (compiled in the
// same translation unit with the same flags), and folded into the step
// slot with the same warp / block minimum and 64-bit atomicMin; the slot
// must hold the dt cap already (rearm_kernel). A minimum does not depend
// on the order, so the dt is the bits the separate kernels give.
//
// Bound by the loads in flight: a thread takes two neighbouring cells, so a
// request is 16 bytes and a source index, read first, is waited for once
// for both (patches and strides are even; 120 us for 29,138 quads of 16x16,
// 478 MB, with one cell a thread, 96 us with two; 6811 quads 31 and 23 us).
#pragma once

#include "stage_kernel.cuh"

namespace amrgpu {

template <int N, class Cand>
__global__ void __launch_bounds__(256) remap_cfl_kernel(const RemapCflArgs a)
{
    constexpr int NN = N * N;
    __shared__ double red[8];
    const CflArgs &c = a.cfl;
    double best = __longlong_as_double((long long)c.scal->slot[c.slot].dt_bits);
    const long long total = (long long)c.nquad * (NN / 2);
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < total;
         p += (long long)gridDim.x * blockDim.x) {
        const int q = (int)(p / (NN / 2));
        const int r = 2 * (int)(p - (long long)q * (NN / 2));
        const int s = a.src[q];
        const bool inject = a.kind[q] == 0;
        double v[2][4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const double *o = a.qold + f * a.stride_old + (long long)s * NN + r;
            double2 w = *reinterpret_cast<const double2 *>(o);
            if (!inject) {
                const double2 w1 = *reinterpret_cast<const double2 *>(o + NN);
                const double2 w2 = *reinterpret_cast<const double2 *>(o + 2 * NN);
                const double2 w3 = *reinterpret_cast<const double2 *>(o + 3 * NN);
                w.x = 0.25 * (w.x + w1.x + w2.x + w3.x);
                w.y = 0.25 * (w.y + w1.y + w2.y + w3.y);
            }
            v[0][f] = w.x;
            v[1][f] = w.y;
            *reinterpret_cast<double2 *>(a.qnew + f * c.stride + (long long)q * NN + r) = w;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double cand = Cand::template candidate<N>(c, q, r + k, v[k]);
            if (cand < best) best = cand;
        }
    }
    best = warp_min(best);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) best = (red[w] < best) ? red[w] : best;
        atomicMin(&c.scal->slot[c.slot].dt_bits, (unsigned long long)__double_as_longlong(best));
    }
}

}  // namespace amrgpu
