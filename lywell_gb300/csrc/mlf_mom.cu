// Dense method-of-moments operator on the GPU (modMoM.f90:85-128 fill,
// MatxVec_MoM modMoM.f90:273-277): the full N x N impedance matrix in FP64,
// filled on the device by the same Z_mn element as the near field, and a
// matvec that streams it once per column where a block's columns are few or the
// matrix small, else once per group of twelve (mlf_split64.cu).  A context made
// with MLF_FLAG_DENSE_MOM holds this operator instead of the octree; CGS,
// excitation and RCS run on it unchanged.  At N = 30720 the matrix is 15 GB, within
// HBM, so it also serves as the exact reference for the MLFMA matvec error.
#include <cuda_runtime.h>

#include <algorithm>

#include "mlf_internal.h"
#include "mlf_fma64.cuh"
#include "mlf_zmn.cuh"

namespace mlf {

#define CK(call)                                             \
    do {                                                     \
        if (!cuda_ok(c, (call), #call)) return MLF_E_CUDA;   \
    } while (0)

// row m per block: Z[m][n] for all n (row-major)
__global__ void k_mom_fill(int N, const double* __restrict__ t_baric, const double* __restrict__ t_baric_sub,
                           const double* __restrict__ p_coord, const int* __restrict__ e_t, const int* __restrict__ e_po,
                           const double* __restrict__ e_long, double w, double w_smue, double c72,
                           double2* __restrict__ Z) {
    const int m = blockIdx.x;
    for (int n = threadIdx.x; n < N; n += blockDim.x)
        Z[(size_t)m * N + n] = zmn_mom(m, n, t_baric, t_baric_sub, p_coord, e_t, e_po, e_long, w, w_smue, c72);
}

// y(m) = sum_n Z[m][n] x(n) for column blockIdx.y: one warp per row, four entries
// a lane in flight, summed in the order of n.  The FP64 pipe bounds it (0.33 ms of
// DFMA at 6750 unknowns, one column): 0.34 ms; one entry in flight, behind a loop
// over four columns, took 1.47 ms.
__global__ void k_mom_gemv(int N, int ld, const double2* __restrict__ Z, const double2* __restrict__ x,
                           double2* __restrict__ y) {
    x += (size_t)blockIdx.y * ld;
    y += (size_t)blockIdx.y * ld;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= N) return;
    const int m = (int)gw;
    const double2 t = warp_sum(dense_terms(lane, 32, N, Z + (size_t)m * N, x));
    if (lane == 0) y[m] = t;
}

int dense_setup(Ctx* c) {
    CK(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    for (int i = 0; i < 8; ++i) CK(cudaEventCreate(&c->ev[i]));
    int st;
    if ((st = upload_geometry(c))) return st;
    const size_t bytes = (size_t)c->N * c->N * sizeof(double2);
    size_t fre = 0, tot = 0;
    CK(cudaMemGetInfo(&fre, &tot));
    if (bytes + ((size_t)1 << 30) > fre) {
        c->err = "dense MoM matrix does not fit in device memory";
        return MLF_E_NOMEM;
    }
    CK(cudaMalloc(&c->dZdense, bytes));
    const double c72 = (double)(1.0f / 72.0f);   // (1./72.) in single precision, as the near field
    k_mom_fill<<<c->N, 256, 0, c->stream>>>(c->N, c->dt_baric, c->dt_baric_sub, c->dp_coord, c->de_t, c->de_po,
                                            c->de_long, c->ph.w, c->ph.w * c->ph.smue, c72, c->dZdense);
    CK(cudaGetLastError());
    if ((st = dense64_setup(c))) return st;
    CK(cudaStreamSynchronize(c->stream));
    return MLF_OK;
}

int dense_matvec(Ctx* c, const double2* x, double2* y, int nrhs, int ld, cudaStream_t s) {
    // blocks of columns go to the digit splits, but for small matrices, where their
    // six launches a group of columns (about 30 us) cost more: 1080 unknowns x 2 is
    // 36 us either way
    if (nrhs > 1 && (double)c->N * c->N * std::min(nrhs, OZ_DENSE_COLS) > 2.5e6)
        return dense64_matvec(c, x, y, nrhs, ld, s);
    const unsigned ctas = (unsigned)(((long long)c->N * 32 + 255) / 256);
    for (int c0 = 0; c0 < nrhs; c0 += 65535)   // a grid has so many rows
        k_mom_gemv<<<dim3(ctas, std::min(nrhs - c0, 65535)), 256, 0, s>>>(c->N, ld, c->dZdense, x + (size_t)c0 * ld,
                                                                          y + (size_t)c0 * ld);
    return cuda_ok(c, cudaGetLastError(), "dense matvec") ? MLF_OK : MLF_E_CUDA;
}

}  // namespace mlf
