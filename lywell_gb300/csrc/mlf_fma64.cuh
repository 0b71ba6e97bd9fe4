// Sums of the FP64 operator in FMAs, one value each: for the kernels that compute
// whole products so and for the digit splits' values that are computed again.
#pragma once

#include <cuda_runtime.h>

namespace mlf {

__device__ __forceinline__ void cmac(double2& acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, acc.x);
    acc.x = fma(-a.y, b.y, acc.x);
    acc.y = fma(a.x, b.y, acc.y);
    acc.y = fma(a.y, b.x, acc.y);
}

// Leaf field of direction q over the bases j0 .. j1 - 1 of a box
__device__ __forceinline__ double2 aggregate_direction(int K2, int j0, int j1, int q, const int* __restrict__ perm,
                                                       const double2* __restrict__ R, const double2* __restrict__ xr) {
    double2 acc = make_double2(0, 0);
    for (int j = j0; j < j1; ++j) cmac(acc, R[(size_t)j * K2 + q], xr[perm[j]]);
    return acc;
}

// The sum over a warp's lanes, in every lane
__device__ __forceinline__ double2 warp_sum(double2 t) {
    double tr = t.x, ti = t.y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tr += __shfl_xor_sync(0xffffffff, tr, o);
        ti += __shfl_xor_sync(0xffffffff, ti, o);
    }
    return make_double2(tr, ti);
}

// Terms first, first + step, ... of y(n) = j facy sum conj(R_j) A_box + sum_near Z x,
// box-sorted basis j = perm^-1(n)
__device__ __forceinline__ double2 receive_near_terms(int first, int step, int K2, int n, const double2* __restrict__ Rj,
                                                      const double2* __restrict__ Ab, const int* __restrict__ ia,
                                                      const int* __restrict__ ja, const double2* __restrict__ Zd,
                                                      const double2* __restrict__ xr, double facy) {
    double sr = 0, si = 0;
    for (int q = first; q < K2; q += step) {
        const double2 a = Rj[q], v = Ab[q];
        sr = fma(a.x, v.x, sr); sr = fma(a.y, v.y, sr);
        si = fma(a.x, v.y, si); si = fma(-a.y, v.x, si);
    }
    double nr = 0, ni = 0;
    for (int q = ia[n] + first; q < ia[n + 1]; q += step) {
        const double2 z = Zd[q];
        const double2 xv = xr[ja[q]];
        nr = fma(xv.x, z.x, nr); nr = fma(-xv.y, z.y, nr);
        ni = fma(xv.x, z.y, ni); ni = fma(xv.y, z.x, ni);
    }
    return make_double2(fma(-facy, si, nr), fma(facy, sr, ni));   // combined before the reduction
}

// Terms first, first + step, ... of row zr of a dense matrix times x, four in flight,
// summed in order
__device__ __forceinline__ double2 dense_terms(int first, int step, int N, const double2* __restrict__ zr,
                                               const double2* __restrict__ x) {
    double ar = 0, ai = 0;
#pragma unroll 4
    for (int n = first; n < N; n += step) {
        const double2 z = zr[n], v = x[n];
        ar = fma(z.x, v.x, ar); ar = fma(-z.y, v.y, ar);
        ai = fma(z.x, v.y, ai); ai = fma(z.y, v.x, ai);
    }
    return make_double2(ar, ai);
}

}  // namespace mlf
