// FP64 near field, leaf aggregation and leaf receive on blocks of columns, on
// the tensor cores, by exact splitting into 8-bit digits (Ozaki, Ogita, Oishi
// and Rump 2012; on FP16 matrix units Mukunoki et al. 2020).
//
// The three are a complex GEMM per leaf box (llenar_campoCyB,
// modMLFMA.f90:1805-1811; MatxVec_MLFMA, :1915-1942):
//   near       y_m = sum_k Z_mk x_k     the box's bases over its near list S,
//                                       which they share; Z complex(4)
//   receive    y_m = sum_k conj(R_mk) A_k   its bases over the 2K directions
//   aggregate  C_q = sum_k R_kq x_k     the directions over its bases
// and the dense method-of-moments operator (MatxVec_MoM, modMoM.f90:273-277) is
// one over all unknowns.
// GB300 does 2 DFMA a clock and SM, which bounds them whatever the number of
// columns; an FP16 product of two integers below 2^8 is exact, and so is its
// FP32 sum.  Both operands become 62-bit integers relative to a power of two
// above the largest value of the row or column, cut into eight signed digits in
// [-128, 127] of weight 2^(8 (7 - i)).  The 36 digit products with i + j <= 7
// are summed per s = i + j in FP32 over 64 real terms: at most 8 * 64 * 2^14 =
// 2^23, exact; then the eight sums are joined in 64-bit integers over all terms,
// and rounded to double once at the end.  What is left out, the products with
// i + j >= 8 foremost, is under 2^-59 a real term (typically 2^-62, of either sign)
// of the bound 2^(er + ec) on the row's and column's largest product.  In the near
// field (and the dense operator) each source k is scaled by a power of two before
// that: x_k to magnitude one (over the block's columns), Z's column k by the
// inverse, so that the bound is near the row's largest term |Z_mk x_k| also where
// x varies over decades.
//
// A column that varies otherwise than its neighbours, or a row whose large entries
// meet small ones of x, can have terms far below that bound.  So each value is
// checked: the top digits' magnitudes are multiplied too (a 37th product), and
// their sum says how large the value's terms are.  A value whose terms' sum is not
// surely 2^-6 of the bound (OZ_COVER) or more, or whose row or column has an Inf
// or a NaN, is computed again in FP64 FMAs (mlf_fma64.cuh): what stands beside a
// column costs time, not digits.
// Error against extended precision over the terms' sum, rms (dense operator of 1920
// unknowns, FMAs -> here): Gaussian columns 7.7e-17 -> 2.4e-17; a column over two
// decades beside them 9.4e-17 -> 5.8e-17 with 21 % of the values computed again, over
// six decades 1.0e-16 -> 9.0e-17 with 68 %.  Of the spheroid's product below, one
// value in 288000 is.
//
// mma.sync keeps each digit sum in the registers of the warp that joins it.
// 12000-RWG spheroid (49 M near entries), 24 columns: the whole product 9.77 ms with
// FMAs, 1.95 ms without the check, 1.96 to 2.02 ms with it.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "mlf_internal.h"
#include "mlf_fma64.cuh"

namespace mlf {

#define CK(call)                                             \
    do {                                                     \
        if (!cuda_ok(c, (call), #call)) return MLF_E_CUDA;   \
    } while (0)

constexpr int OZ_D = 8;            // digits
constexpr int OZ_R = 64;           // rows (bases of one box) per CTA
constexpr int OZ_K = 32;           // bases of S per step: 64 real terms
constexpr int OZ_PITCH = 4 * OZ_K + 16;                    // bytes of a row of 64 FP16, padded: ldmatrix without conflicts
constexpr int OZ_ABYTES = OZ_D * OZ_R * OZ_PITCH;          // Z digits  [digit][row][term]
constexpr int OZ_BBYTES = OZ_D * 2 * OZ_C * OZ_PITCH;      // x digits  [digit][real column][term]
constexpr int OZ_STAGE = OZ_ABYTES + OZ_BBYTES;
constexpr int OZ_SMEM = 2 * OZ_STAGE + (OZ_R + OZ_C) * 4;
constexpr int OZ_WARPS = 12;       // 4 tiles of 16 rows x 3 of 8 real columns
constexpr int OZ_THREADS = 32 * OZ_WARPS;
constexpr int OZ_WR = (OZ_R + OZ_WARPS - 1) / OZ_WARPS;   // rows that a warp converts
static_assert(OZ_C == OZ_WARPS && 2 * OZ_C == 8 * (OZ_WARPS / 4), "a warp converts one column and multiplies one tile");

// |v| < 2^e to an integer below 2^62, truncated: v = m 2^(e - 62)
__device__ __forceinline__ long long oz_fix(unsigned long long m62, int t, uint32_t sign) {
    const long long m = (long long)(m62 >> min(t, 63));
    return sign ? -m : m;
}
__device__ __forceinline__ long long oz_fix(float v, int e) {
    const uint32_t b = __float_as_uint(v);
    const int ef = (b >> 23) & 0xff;
    const uint32_t mant = (b & 0x7fffffu) | (ef ? 0x800000u : 0u);
    return oz_fix((unsigned long long)mant << 38, e + 126 - max(ef, 1), b >> 31);
}
__device__ __forceinline__ long long oz_fix(double v, int e) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int ef = (int)(b >> 52) & 0x7ff;
    const unsigned long long mant = (b & 0xfffffffffffffull) | (ef ? 0x10000000000000ull : 0ull);
    return oz_fix(mant << 9, e + 1022 - max(ef, 1), (uint32_t)(b >> 63));
}

// exponent e with |v| < 2^e of the larger of two magnitudes, OZ_ZERO for zeros,
// OZ_BAD for an Inf or a NaN
constexpr int OZ_ZERO = -100000, OZ_BAD = 100000;
// With others added or taken off: of a sum, and its mark for the check below
__device__ __forceinline__ bool oz_zero(int e) { return e < OZ_ZERO / 2; }
__device__ __forceinline__ bool oz_bad(int e) { return e > OZ_BAD / 2; }
__device__ __forceinline__ int oz_exp(float2 v) {
    const uint32_t m = max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu);
    const int ef = (int)(m >> 23);
    return m == 0 ? OZ_ZERO : ef == 0xff ? OZ_BAD : max(ef, 1) - 126;
}
__device__ __forceinline__ int oz_exp(double2 v) {
    const uint32_t m = max((uint32_t)__double2hiint(v.x) & 0x7fffffffu, (uint32_t)__double2hiint(v.y) & 0x7fffffffu);
    const int ef = (int)(m >> 20);
    if (m == 0 && (__double2loint(v.x) | __double2loint(v.y)) == 0) return OZ_ZERO;
    return ef == 0x7ff ? OZ_BAD : max(ef, 1) - 1022;
}

// sexp[n] = exponent of x's row n over the columns where it is finite (a column
// that is not is marked by its own exponent; its entries tell the others nothing),
// the smallest number's where it is zero; *nredo = 0 and, where given, cexp = OZ_ZERO
__global__ void k_row_exp(int N, int nrhs, int ld, const double2* __restrict__ x, int* __restrict__ sexp,
                          int* __restrict__ nredo, int* __restrict__ cexp) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    if (n == 0) *nredo = 0;
    if (cexp)
        for (int c = n; c < nrhs; c += N) cexp[c] = OZ_ZERO;
    int e = OZ_ZERO;
    for (int c = 0; c < nrhs; ++c) {
        const int v = oz_exp(x[(size_t)c * ld + n]);
        if (v != OZ_BAD) e = max(e, v);
    }
    sexp[n] = max(e, -1021);
}

// rexp[pos] = exponent of row perm[pos] of Z 2^sexp; a warp per row
__global__ void k_near_exp(int N, const int* __restrict__ perm, const int* __restrict__ ia, const int* __restrict__ ja,
                           const float2* __restrict__ Z, const int* __restrict__ sexp, int* __restrict__ rexp) {
    const int pos = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (pos >= N) return;
    const int n = perm[pos], q1 = ia[n + 1];
    int e = OZ_ZERO;
#pragma unroll 4
    for (int q = ia[n] + lane; q < q1; q += 32) e = max(e, oz_exp(Z[q]) + sexp[ja[q]]);
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) rexp[pos] = e;
}

enum { OZ_NEAR = 0, OZ_RECEIVE = 1, OZ_AGGREGATE = 2, OZ_DENSE = 3 };

// cexp[box * nrhs + c] = exponent of column c of the box's right-hand operand:
// x 2^-sexp over the near list, the field A over its 2K directions, or x over
// the box's bases; a CTA per pair
template <int MODE>
__global__ void k_col_exp(int nrhs, int ld, int K2, const int* __restrict__ box_ptr, const int* __restrict__ perm,
                          const int* __restrict__ ia, const int* __restrict__ ja, const double2* __restrict__ x,
                          const int* __restrict__ sexp, int* __restrict__ cexp, int* __restrict__ redo) {
    const int b = blockIdx.x / nrhs, c = blockIdx.x % nrhs;
    __shared__ int top;
    if (threadIdx.x == 0) {
        top = OZ_ZERO;
        if (MODE == OZ_AGGREGATE) redo[blockIdx.x] = 0;
    }
    __syncthreads();
    int e = OZ_ZERO;
    if (MODE == OZ_NEAR) {
        const int n = perm[box_ptr[b]], q1 = ia[n + 1];
        for (int q = ia[n] + threadIdx.x; q < q1; q += blockDim.x)
            e = max(e, oz_exp(x[(size_t)c * ld + ja[q]]) - sexp[ja[q]]);
    } else if (MODE == OZ_RECEIVE) {
        for (int q = threadIdx.x; q < K2; q += blockDim.x) e = max(e, oz_exp(x[(size_t)blockIdx.x * K2 + q]));
    } else {
        for (int q = box_ptr[b] + threadIdx.x; q < box_ptr[b + 1]; q += blockDim.x)
            e = max(e, oz_exp(x[(size_t)c * ld + perm[q]]));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&top, e);
    __syncthreads();
    if (threadIdx.x == 0) cexp[blockIdx.x] = top;
}

// exponents of the patterns, once per context: of each basis over the directions
// (a warp per basis), and of each box's directions over its bases
__global__ void k_pattern_exp(int N, int K2, const double2* __restrict__ R, int* __restrict__ rexp) {
    const int pos = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (pos >= N) return;
    int e = OZ_ZERO;
    for (int q = lane; q < K2; q += 32) e = max(e, oz_exp(R[(size_t)pos * K2 + q]));
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) rexp[pos] = e;
}
// ... a CTA per box and 32 directions, its warps over the bases (12000-RWG spheroid, 32
// boxes: 30 us; a CTA a box, 390)
__global__ void __launch_bounds__(256) k_direction_exp(int K2, const int* __restrict__ box_ptr,
                                                       const double2* __restrict__ R, int* __restrict__ qexp) {
    __shared__ int top[8][32];
    const int b = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = blockIdx.y * 32 + lane;
    int e = OZ_ZERO;
    if (q < K2)
#pragma unroll 4
        for (int t = box_ptr[b] + warp; t < box_ptr[b + 1]; t += 8) e = max(e, oz_exp(R[(size_t)t * K2 + q]));
    top[warp][lane] = e;
    __syncthreads();
    if (warp || q >= K2) return;
    for (int w = 1; w < 8; ++w) e = max(e, top[w][lane]);
    qexp[(size_t)b * K2 + q] = e;
}

// The digits of (re, im) as FP16 pairs, most significant first: with 128 added
// to every digit the bytes of the integer are the biased digits; 0x6400 | byte
// is 1024 + byte in FP16.
__device__ __forceinline__ void oz_digits(long long re, long long im, uint32_t (&d)[OZ_D]) {
    const unsigned long long bias = 0x8080808080808080ull;
    const unsigned long long r = (unsigned long long)re + bias, i = (unsigned long long)im + bias;
    const uint32_t w[4] = {(uint32_t)(r >> 32), (uint32_t)(i >> 32), (uint32_t)r, (uint32_t)i};
    const __half2 off = __float2half2_rn(-1152.f);
#pragma unroll
    for (int q = 0; q < OZ_D; ++q) {
        const int byte = 3 - (q & 3);   // of the high words, then of the low ones
        const uint32_t x = (__byte_perm(w[q / 4 * 2], w[q / 4 * 2 + 1], byte | (4 + byte) << 8) & 0x00ff00ffu) | 0x64006400u;
        const __half2 h = __hadd2(*reinterpret_cast<const __half2*>(&x), off);
        d[q] = *reinterpret_cast<const uint32_t*>(&h);
    }
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 2^(er + ec - 68) (hi 2^32 + lo): digit i weighs 2^(e - 62 + 8 (7 - i)), the sum
// s of hi and lo 2^(8 (7 - s)) of 2^(er + ec - 124 + 56)
__device__ __forceinline__ double oz_value(long long hi, long long lo, int er, int ec) {
    return ldexp(fma((double)hi, 4294967296.0, (double)lo), er + ec - 68);
}

// Dense operator.  bexp[row * nblk + b] = exponent of the row over the 32 unknowns
// of block b, once per context; a warp per row
__global__ void k_dense_block_exp(int N, int nblk, const double2* __restrict__ Z, short* __restrict__ bexp) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= N) return;
#pragma unroll 4
    for (int b = 0; b < nblk; ++b) {
        const int k = 32 * b + lane;
        const int e = __reduce_max_sync(0xffffffffu, k < N ? oz_exp(Z[(size_t)row * N + k]) : OZ_ZERO);
        if (lane == 0) bexp[(size_t)row * nblk + b] = (short)min(max(e, -2000), 2000);   // 2000: not finite
    }
}
// bmax[b] = largest sexp of block b; cexp[c] = exponent of column c of x 2^-sexp
__global__ void k_dense_col_exp(int N, int nrhs, int ld, int nblk, const double2* __restrict__ x,
                                const int* __restrict__ sexp, int* __restrict__ bmax, int* __restrict__ cexp) {
    const int lane = threadIdx.x & 31;
    for (int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nblk; b += (gridDim.x * blockDim.x) >> 5) {
        const int k = 32 * b + lane;
        const int s = k < N ? sexp[k] : OZ_ZERO, e = __reduce_max_sync(0xffffffffu, s);
        if (lane == 0) bmax[b] = e;
        for (int c = 0; c < nrhs; ++c) {
            const int v = __reduce_max_sync(0xffffffffu, k < N ? oz_exp(x[(size_t)c * ld + k]) - s : OZ_ZERO);
            if (lane == 0) atomicMax(&cexp[c], v);
        }
    }
}
// rexp[row] = bound of the exponent of row of Z 2^sexp, by blocks
__global__ void k_dense_row_exp(int N, int nblk, const short* __restrict__ bexp, const int* __restrict__ bmax,
                                int* __restrict__ rexp) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= N) return;
    int e = OZ_ZERO;
    for (int b = lane; b < nblk; b += 32) {
        const int v = bexp[(size_t)row * nblk + b];
        e = max(e, v == 2000 ? OZ_BAD : v + bmax[b]);
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) rexp[row] = e;
}
// The check of a value: cover = sum over the real terms of its two parts of the
// product of the top digits' magnitudes, parts of the terms added up.  A top digit
// d stands for a magnitude of (|d| - 0.51) 2^-6 or more of its operand's bound, so a
// cover of 512 surely means complex terms of 512 / 2 / 4 * 2^-12 = 2^-6 of the value's
// bound in sum (a part that is small beside the other is off by what that one allows).
constexpr float OZ_COVER = 512.f, OZ_SURE = 1e30f;
__device__ __forceinline__ float oz_cover(float c, int er, int ec) {
    if (oz_bad(er) || oz_bad(ec)) return -OZ_SURE;
    return oz_zero(er) || oz_zero(ec) ? OZ_SURE : c;   // exactly zero
}

// list[(*n)++] = v of each active lane
__device__ __forceinline__ void oz_append(int* n, unsigned* list, unsigned v) {
    const unsigned on = __activemask(), lane = threadIdx.x & 31;
    const int first = __ffs(on) - 1;
    int base = 0;
    if ((int)lane == first) base = atomicAdd(n, __popc(on));
    base = __shfl_sync(on, base, first);
    list[base + __popc(on & ((1u << lane) - 1))] = v;
}

// y = sum of the parts, in order
__global__ void k_sum_parts(int N, int nrhs, int ld, int nsplit, const double2* __restrict__ ws,
                            const float* __restrict__ cov, double2* __restrict__ y, int* __restrict__ nredo,
                            unsigned* __restrict__ redo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (i >= N) return;
    double2 t = make_double2(0, 0);
    float g = 0.f;
    for (int p = 0; p < nsplit; ++p) {
        const size_t at = ((size_t)p * nrhs + c) * N + i;
        const double2 v = ws[at];
        t.x += v.x;
        t.y += v.y;
        g += cov[at];
    }
    y[(size_t)c * ld + i] = t;
    if (g < OZ_COVER) oz_append(nredo, redo, (unsigned)c * N + i);
}

// Values computed again in FMAs.  Leaf fields: CTA (box, column), where one of its
// directions asks for it
__global__ void k_redo_aggregate(int K2, int nrhs, int ld, const int* __restrict__ redo,
                                 const int* __restrict__ box_ptr, const int* __restrict__ perm,
                                 const double2* __restrict__ R, const double2* __restrict__ x, double2* __restrict__ C) {
    if (!redo[blockIdx.x]) return;
    const int b = blockIdx.x / nrhs, r = blockIdx.x % nrhs;
    for (int q = threadIdx.x; q < K2; q += blockDim.x)
        C[(size_t)blockIdx.x * K2 + q] =
            aggregate_direction(K2, box_ptr[b], box_ptr[b + 1], q, perm, R, x + (size_t)r * ld);
}
// The listed values v: store(v, sum of terms(v, first, step) over first = 0 .. step - 1).
// A warp each, or, while there are no more of them than CTAs, a CTA each: one row's
// chain of FP64 FMAs is the time then (one row of 4100 terms 18 us, with a warp 71).
constexpr int OZ_REDO_T = 256;
template <class Terms, class Store>
__device__ __forceinline__ void redo_listed(int n, const unsigned* __restrict__ redo, Terms terms, Store store) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (n <= (int)gridDim.x) {
        __shared__ double2 part[OZ_REDO_T / 32];
        if ((int)blockIdx.x >= n) return;
        const unsigned v = redo[blockIdx.x];
        const double2 t = warp_sum(terms(v, threadIdx.x, OZ_REDO_T));
        if (lane == 0) part[warp] = t;
        __syncthreads();
        if (threadIdx.x == 0) {
            double2 s = part[0];
            for (int w = 1; w < OZ_REDO_T / 32; ++w) {
                s.x += part[w].x;
                s.y += part[w].y;
            }
            store(v, s);
        }
        return;
    }
    for (int k = blockIdx.x * (OZ_REDO_T / 32) + warp; k < n; k += gridDim.x * (OZ_REDO_T / 32)) {
        const unsigned v = redo[k];
        const double2 t = warp_sum(terms(v, lane, 32));
        if (lane == 0) store(v, t);
    }
}
// y of the listed (column, box-sorted basis)
__global__ void __launch_bounds__(OZ_REDO_T)
k_redo_receive_near(int K2, int N, int nrhs, int ld, const int* __restrict__ nredo, const unsigned* __restrict__ redo,
                    const int* __restrict__ perm, const int* __restrict__ box_of_sorted, const double2* __restrict__ R,
                    const double2* __restrict__ A, const int* __restrict__ ia, const int* __restrict__ ja,
                    const double2* __restrict__ Zd, const double2* __restrict__ x, double facy, double2* __restrict__ y) {
    redo_listed(*nredo, redo,
                [&](unsigned v, int first, int step) {
                    const int r = v / N, j = v % N;
                    return receive_near_terms(first, step, K2, perm[j], R + (size_t)j * K2,
                                              A + ((size_t)box_of_sorted[j] * nrhs + r) * K2, ia, ja, Zd,
                                              x + (size_t)r * ld, facy);
                },
                [&](unsigned v, double2 t) { y[(size_t)(v / N) * ld + perm[v % N]] = t; });
}
// y of the listed (column, row) of the dense operator
__global__ void __launch_bounds__(OZ_REDO_T) k_redo_dense(int N, int ld, const int* __restrict__ nredo,
                                                          const unsigned* __restrict__ redo,
                                                          const double2* __restrict__ Z, const double2* __restrict__ x,
                                                          double2* __restrict__ y) {
    redo_listed(*nredo, redo,
                [&](unsigned v, int first, int step) {
                    return dense_terms(first, step, N, Z + (size_t)(v % N) * N, x + (size_t)(v / N) * ld);
                },
                [&](unsigned v, double2 t) { y[(size_t)(v / N) * ld + v % N] = t; });
}

struct OzArgs {
    int N, nrhs, ld, K2;                // K2 = 2K, the leaf's samples of both polarisations
    const int2* tiles;                  // (box, first row)
    const int *box_ptr, *perm, *ia, *ja;
    const float2* Z;
    const double2 *R, *x;               // R: patterns, or the dense matrix; x: right-hand operand (receive: the field A)
    const int *sexp, *rexp, *cexp;      // exponents of sources (near), rows and columns
    double2* out;                       // near: [split][col][box-sorted place]; receive: y; aggregate: the field C
    const double2* near;                // receive: the near field's parts
    float* cov;                        // near: the parts' covers, as out (receive: read)
    int* nredo;                         // receive: values to compute again, and their list
    unsigned* redo;
    int* redo_box;                      // aggregate: (box, column) to compute again
    int nsplit;
    double facy;
};

template <int MODE> struct OzLeft { typedef double2 T; };
template <> struct OzLeft<OZ_NEAR> { typedef float2 T; };

// blockIdx.x = (row tile, block of 12 columns), .y = part of the near list.  While one step's
// digits are multiplied the next step's are made in the other stage, half of the
// warps beginning with the one, half with the other, and the values of the step
// after are on their way to registers.
template <int MODE>
__global__ void __launch_bounds__(OZ_THREADS, 1) k_split64(const OzArgs g) {
    typedef typename OzLeft<MODE>::T ZT;
    extern __shared__ __align__(16) unsigned char oz_smem[];
    int* er = reinterpret_cast<int*>(oz_smem + 2 * OZ_STAGE);   // exponent of each row
    int* ec = er + OZ_R;                                         // ... and of each column
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nqt = (g.K2 + OZ_R - 1) / OZ_R;
    const int ncb = (g.nrhs + OZ_C - 1) / OZ_C, tile = blockIdx.x / ncb;
    const int2 tl = MODE == OZ_DENSE ? make_int2(0, tile * OZ_R) : MODE == OZ_AGGREGATE ? make_int2(tile / nqt, tile % nqt * OZ_R) : g.tiles[tile];
    const int b0 = MODE == OZ_DENSE ? 0 : g.box_ptr[tl.x], nb = MODE == OZ_DENSE ? g.N : g.box_ptr[tl.x + 1] - b0;
    const int p0 = b0 + tl.y;                                    // near, receive: rows p0 .. p0 + nr - 1
    const int nr = min(OZ_R, (MODE == OZ_AGGREGATE ? g.K2 : nb) - tl.y);
    const int c0 = blockIdx.x % ncb * OZ_C, nc = min(OZ_C, g.nrhs - c0);
    const int s0 = MODE == OZ_NEAR ? g.ia[g.perm[b0]] : 0;
    const int len = MODE == OZ_NEAR ? g.ia[g.perm[b0] + 1] - s0 : MODE == OZ_RECEIVE ? g.K2 : nb;
    const int nstep = (len + OZ_K - 1) / OZ_K;
    const int k0 = (int)((long long)nstep * blockIdx.y / gridDim.y) * OZ_K;
    const int k1 = min(len, (int)((long long)nstep * (blockIdx.y + 1) / gridDim.y) * OZ_K);
    const int* rexp = g.rexp + (MODE == OZ_AGGREGATE ? (size_t)tl.x * g.K2 + tl.y : (size_t)p0);
    if (tid < OZ_R) er[tid] = tid < nr ? rexp[tid] : OZ_ZERO;
    if (tid < OZ_C) ec[tid] = tid < nc ? g.cexp[(size_t)tl.x * g.nrhs + c0 + tid] : OZ_ZERO;
    __syncthreads();
    // warp w converts the rows w, w + 12, ... and the column w
    const ZT* zrow[OZ_WR];
#pragma unroll
    for (int r = 0; r < OZ_WR; ++r) {
        const int row = min(warp + OZ_WARPS * r, nr - 1);
        if constexpr (MODE == OZ_NEAR) zrow[r] = g.Z + g.ia[g.perm[p0 + row]];
        else if constexpr (MODE == OZ_RECEIVE) zrow[r] = g.R + (size_t)(p0 + row) * g.K2;
        else if constexpr (MODE == OZ_DENSE) zrow[r] = g.R + (size_t)(p0 + row) * g.N;
        else zrow[r] = g.R + (size_t)b0 * g.K2 + tl.y + row;
    }
    const int col = c0 + min(warp, nc - 1);
    const double2* xc = MODE == OZ_RECEIVE ? g.x + ((size_t)tl.x * g.nrhs + col) * g.K2 : g.x + (size_t)col * g.ld;
    auto source = [&](int k) {   // of the right-hand operand; k includes the lane
        if (k >= k1) return -1;
        return MODE == OZ_NEAR ? g.ja[s0 + k] : MODE == OZ_AGGREGATE ? g.perm[b0 + k] : k;
    };
    auto shift = [&](int j) { return (MODE == OZ_NEAR || MODE == OZ_DENSE) && j >= 0 ? g.sexp[j] : 0; };
    ZT z[OZ_WR];
    double2 xv;
    auto load = [&](int k, int j) {
#pragma unroll
        for (int r = 0; r < OZ_WR; ++r) {
            z[r].x = z[r].y = 0;
            if (j >= 0 && warp + OZ_WARPS * r < nr) {
                z[r] = zrow[r][MODE == OZ_AGGREGATE ? (size_t)k * g.K2 : (size_t)k];
                if (MODE == OZ_RECEIVE) z[r].y = -z[r].y;
            }
        }
        xv = j >= 0 && warp < nc ? xc[j] : make_double2(0, 0);
    };
    // the loaded values to digits in stage `st`
    auto convert = [&](unsigned char* st, int se) {
        uint32_t d[OZ_D];
#pragma unroll
        for (int r = 0; r < OZ_WR; ++r) {
            const int row = warp + OZ_WARPS * r;
            if (row >= OZ_R) break;
            const int e = er[row] - se;
            oz_digits(oz_fix(z[r].x, e), oz_fix(z[r].y, e), d);
#pragma unroll
            for (int q = 0; q < OZ_D; ++q)
                *reinterpret_cast<uint32_t*>(st + (q * OZ_R + row) * OZ_PITCH + lane * 4) = d[q];
        }
        const int e = ec[warp] + se;
        oz_digits(oz_fix(xv.x, e), oz_fix(xv.y, e), d);
#pragma unroll
        for (int q = 0; q < OZ_D; ++q) {   // (Re x, -Im x) for Re y, (Im x, Re x) for Im y
            unsigned char* row = st + OZ_ABYTES + (q * 2 * OZ_C + 2 * warp) * OZ_PITCH + lane * 4;
            *reinterpret_cast<uint32_t*>(row) = d[q] ^ 0x80000000u;
            *reinterpret_cast<uint32_t*>(row + OZ_PITCH) = __byte_perm(d[q], 0, 0x1032);
        }
    };
    const int mt = warp & 3, nt = warp >> 2;   // row tile, column tile
    const bool mine = mt * 16 < nr && nt * 4 < nc;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(oz_smem);
    const uint32_t a_addr = base + (mt * 16 + (lane & 15)) * OZ_PITCH + (lane >> 4) * 16;
    const uint32_t b_addr = base + OZ_ABYTES + (lane >> 4) * (2 * OZ_C * OZ_PITCH) +
                            (nt * 8 + (lane & 7)) * OZ_PITCH + ((lane >> 3) & 1) * 16;
    long long hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
    float cover[4] = {0.f, 0.f, 0.f, 0.f};
    auto products = [&](uint32_t off) {
        float acc[OZ_D][4];
#pragma unroll
        for (int s = 0; s < OZ_D; ++s)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[s][q] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 2 * OZ_K / 16; ++ks) {
            uint32_t b[OZ_D / 2][4];   // digits 2 p and 2 p + 1
#pragma unroll
            for (int p = 0; p < OZ_D / 2; ++p) ldsm4(b[p], b_addr + off + 2 * p * (2 * OZ_C * OZ_PITCH) + ks * 32);
#pragma unroll
            for (int i = 0; i < OZ_D; ++i) {
                uint32_t a[4];
                ldsm4(a, a_addr + off + i * (OZ_R * OZ_PITCH) + ks * 32);
                if (i == 0) {   // the top digits' magnitudes
                    constexpr uint32_t M = 0x7fff7fffu;
                    const uint32_t m[4] = {a[0] & M, a[1] & M, a[2] & M, a[3] & M};
                    mma_f16(cover, m, b[0][0] & M, b[0][1] & M);
                }
#pragma unroll
                for (int j = 0; i + j < OZ_D; ++j)
                    mma_f16(acc[i + j], a, b[j / 2][2 * (j & 1)], b[j / 2][2 * (j & 1) + 1]);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            long long v[OZ_D];
#pragma unroll
            for (int s = 0; s < OZ_D; ++s) v[s] = __float2int_rn(acc[s][q]);
            hi[q] += v[0] * 16777216 + v[1] * 65536 + v[2] * 256 + v[3];
            lo[q] += v[4] * 16777216 + v[5] * 65536 + v[6] * 256 + v[7];
        }
    };
    int j = source(k0 + lane), jn = source(k0 + OZ_K + lane);   // of the next step to convert, and the one after
    load(k0 + lane, j);
    int se = shift(j);
    convert(oz_smem, se);
    auto turn = [&](int k) {   // the loads that the following steps need
        j = jn;
        load(k + lane, j);
        se = shift(j);
        jn = source(k + OZ_K + lane);
    };
    turn(k0 + OZ_K);
    int st = 0;
    for (int kb = k0; kb < k1; kb += OZ_K, st ^= 1) {
        __syncthreads();   // this step's digits are there, the other stage has been multiplied
        auto next = [&]() {
            if (kb + OZ_K >= k1) return;
            convert(oz_smem + (st ^ 1) * OZ_STAGE, se);
            turn(kb + 2 * OZ_K);
        };
        if ((warp >> 2) & 1) next();
        if (mine) products(st * OZ_STAGE);
        if (!((warp >> 2) & 1)) next();
    }
    if (!mine) return;
    const int cc = nt * 4 + (lane & 3);
    if (cc >= nc) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = mt * 16 + 8 * h + (lane >> 2);
        if (row >= nr) continue;
        const int e = er[row], f = ec[cc];
        double2 v = make_double2(oz_value(hi[2 * h], lo[2 * h], e, f), oz_value(hi[2 * h + 1], lo[2 * h + 1], e, f));
        const float cv = oz_cover(cover[2 * h] + cover[2 * h + 1], e, f);
        if (MODE == OZ_NEAR || MODE == OZ_DENSE) {
            const size_t at = ((size_t)blockIdx.y * g.nrhs + c0 + cc) * g.N + p0 + row;
            g.out[at] = v;
            g.cov[at] = cv;
        } else if (MODE == OZ_AGGREGATE) {
            g.out[((size_t)tl.x * g.nrhs + c0 + cc) * g.K2 + tl.y + row] = v;
            if (cv < OZ_COVER) g.redo_box[(size_t)tl.x * g.nrhs + c0 + cc] = 1;
        } else {   // y = j facy v + near
            double2 w = make_double2(0, 0);
            float cn = 0.f;
            for (int p = 0; p < g.nsplit; ++p) {
                const size_t at = ((size_t)p * g.nrhs + c0 + cc) * g.N + p0 + row;
                const double2 t = g.near[at];
                w.x += t.x;
                w.y += t.y;
                cn += g.cov[at];
            }
            g.out[(size_t)(c0 + cc) * g.ld + g.perm[p0 + row]] = make_double2(fma(-g.facy, v.y, w.x), fma(g.facy, v.x, w.y));
            if (cv < OZ_COVER || cn < OZ_COVER) oz_append(g.nredo, g.redo, (unsigned)(c0 + cc) * g.N + p0 + row);
        }
    }
}

static float* oz_covers(const Ctx* c) { return reinterpret_cast<float*>(c->doz_ws + c->oz_cap.sums); }

// CTAs that go through a list of values to compute again
constexpr int OZ_REDO_CTAS = 8;   // per SM

static int near64_split(const Ctx* c, int nrhs) { return oz_split(c->noz_tiles, c->nsm, nrhs, c->dense); }

// workspace for blocks of up to nrhs columns, with `fixed` exponents beside it and
// `per_col` more a column
static int oz_workspace(Ctx* c, int nrhs, size_t fixed, size_t per_col) {
    const OzSizes need = oz_sizes(c->noz_tiles, c->nsm, c->N, c->dense, fixed, per_col, nrhs);
    if (!oz_short(c->oz_cap, need)) return MLF_OK;
    if (c->doz_ws) cudaFree(c->doz_ws);
    c->doz_ws = nullptr;
    c->doz_exp = nullptr;
    const OzSizes grown{std::max(c->oz_cap.sums, need.sums), std::max(c->oz_cap.exps, need.exps)};
    c->oz_cap = OzSizes();
    // one allocation: sums, their covers, exponents
    CK(cudaMalloc(&c->doz_ws, grown.sums * (sizeof(double2) + sizeof(float)) + grown.exps * sizeof(int)));
    c->oz_cap = grown;
    c->doz_exp = reinterpret_cast<int*>(oz_covers(c) + grown.sums);
    return MLF_OK;
}

// Where the products run here: a CTA's tile is 64 rows of one box by 12 columns,
// so boxes and blocks must fill it to some part.  Whole products in us, FP64 FMAs
// against here, by bases per box x columns, of bodies of 7680 to 48000 unknowns:
// 4.3 x 24: 21801, 24565; 11.0 x 12: 14051, 13987; 15.5 x 6: 2830, 2915; x 8: 3736,
// 3548; 21.9 x 4: 4118, 4106; x 6: 6061, 5549; 37.3 x 2: 1194, 1351; x 4: 2119, 1703; 41.7 x
// 3: 509, 443; 240 x 2: 639, 421.  One column stays with the FMAs, whose order of
// sums single solves keep.
bool split64_on(const Ctx* c, int nrhs) {
    const long long nb = (long long)c->box_ptr.size() - 1;
    return nrhs >= 2 && c->N >= 12 * nb && (long long)c->N * nrhs >= 112 * nb;
}

// The tile list and the patterns' exponents (once per context), and the
// workspace, grown so that a smaller block never needs more (a caller may
// capture it).
int split64_ready(Ctx* c, int nrhs) {
    const size_t nb = c->box_ptr.size() - 1, K2 = 2 * (size_t)c->lv[c->nlev].K;
    if (!c->doz_tiles) {
        std::vector<int2> t;
        for (size_t b = 0; b < nb; ++b)
            for (int r = 0; r < c->box_ptr[b + 1] - c->box_ptr[b]; r += OZ_R) t.push_back(make_int2((int)b, r));
        CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, c->dev));
        // limits of the kernels, the same for every context
        CK(cudaFuncSetAttribute(k_split64<OZ_NEAR>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
        CK(cudaFuncSetAttribute(k_split64<OZ_RECEIVE>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
        CK(cudaFuncSetAttribute(k_split64<OZ_AGGREGATE>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
        int2* d = nullptr;   // the tiles, then the exponents
        CK(cudaMalloc(&d, t.size() * sizeof(int2) + (c->N + nb * K2) * sizeof(int)));
        int* pat = reinterpret_cast<int*>(d + t.size());
        k_pattern_exp<<<(c->N + 7) / 8, 256, 0, c->stream>>>(c->N, (int)K2, c->dR, pat);
        k_direction_exp<<<dim3((unsigned)nb, (unsigned)(K2 + 31) / 32), 256, 0, c->stream>>>((int)K2, c->dbox_ptr, c->dR, pat + c->N);
        if (!cuda_ok(c, cudaGetLastError(), "pattern exponents") ||
            !cuda_ok(c, cudaMemcpy(d, t.data(), t.size() * sizeof(int2), cudaMemcpyHostToDevice), "tiles") ||
            !cuda_ok(c, cudaStreamSynchronize(c->stream), "pattern exponents")) {   // products may run on another stream
            cudaFree(d);
            return MLF_E_CUDA;
        }
        c->doz_tiles = d;
        c->doz_pat = pat;
        c->noz_tiles = (int)t.size();
    }
    return oz_workspace(c, nrhs, 2 * (size_t)c->N + 1, 2 * nb + c->N);
}

static OzArgs oz_args(const Ctx* c, int nrhs, int ld) {
    OzArgs g{};
    g.N = c->N; g.nrhs = nrhs; g.ld = ld; g.K2 = 2 * c->lv[c->nlev].K;
    g.tiles = c->doz_tiles;
    g.box_ptr = c->dbox_ptr; g.perm = c->dperm; g.ia = c->dia; g.ja = c->dja;
    g.Z = c->dZ; g.R = c->dR;
    return g;
}

// The parts of doz_exp: exponents of sources, rows and columns, values to compute
// again (a flag a box and column, and a list with its length)
struct OzExps {
    int *sexp, *rexp, *nredo, *cexp, *redo_box;
    unsigned* redo;
};
static OzExps oz_exps(const Ctx* c, size_t nb, int nrhs) {
    OzExps e;
    e.sexp = c->doz_exp;
    e.rexp = e.sexp + c->N;
    e.nredo = e.rexp + c->N;
    e.cexp = e.nredo + 1;
    e.redo_box = e.cexp + nb * nrhs;
    e.redo = reinterpret_cast<unsigned*>(e.redo_box + nb * nrhs);
    return e;
}

// C (leaf fields) = R^T x
int split64_aggregate(Ctx* c, const double2* x, int nrhs, int ld, double2* C, cudaStream_t s) {
    const int nb = (int)c->box_ptr.size() - 1;
    OzArgs g = oz_args(c, nrhs, ld);
    const OzExps e = oz_exps(c, nb, nrhs);
    k_col_exp<OZ_AGGREGATE><<<nb * nrhs, 128, 0, s>>>(nrhs, ld, g.K2, g.box_ptr, g.perm, g.ia, g.ja, x, nullptr, e.cexp,
                                                      e.redo_box);
    g.x = x; g.rexp = c->doz_pat + c->N; g.cexp = e.cexp; g.out = C; g.redo_box = e.redo_box;
    k_split64<OZ_AGGREGATE><<<(unsigned)((size_t)nb * ((g.K2 + OZ_R - 1) / OZ_R) * ((nrhs + OZ_C - 1) / OZ_C)), OZ_THREADS,
                              OZ_SMEM, s>>>(g);
    k_redo_aggregate<<<nb * nrhs, 256, 0, s>>>(g.K2, nrhs, ld, e.redo_box, g.box_ptr, g.perm, g.R, x, C);
    return cuda_ok(c, cudaGetLastError(), "aggregation (split)") ? MLF_OK : MLF_E_CUDA;
}

// y = Z_near x + j facy conj(R) A
int split64_receive_near(Ctx* c, const double2* x, const double2* A, double facy, int nrhs, int ld, double2* y,
                         cudaStream_t s) {
    const int nb = (int)c->box_ptr.size() - 1, ncb = (nrhs + OZ_C - 1) / OZ_C;
    OzArgs g = oz_args(c, nrhs, ld);
    const OzExps e = oz_exps(c, nb, nrhs);
    k_row_exp<<<(c->N + 255) / 256, 256, 0, s>>>(c->N, nrhs, ld, x, e.sexp, e.nredo, nullptr);
    k_near_exp<<<(c->N + 7) / 8, 256, 0, s>>>(c->N, c->dperm, c->dia, c->dja, c->dZ, e.sexp, e.rexp);
    k_col_exp<OZ_NEAR><<<nb * nrhs, 256, 0, s>>>(nrhs, ld, g.K2, g.box_ptr, g.perm, g.ia, g.ja, x, e.sexp, e.cexp,
                                                 nullptr);
    const int nsplit = near64_split(c, nrhs);
    g.x = x; g.sexp = e.sexp; g.rexp = e.rexp; g.cexp = e.cexp; g.out = c->doz_ws; g.cov = oz_covers(c);
    k_split64<OZ_NEAR><<<dim3(ncb * c->noz_tiles, nsplit), OZ_THREADS, OZ_SMEM, s>>>(g);
    k_col_exp<OZ_RECEIVE><<<nb * nrhs, 128, 0, s>>>(nrhs, ld, g.K2, g.box_ptr, g.perm, g.ia, g.ja, A, nullptr, e.cexp,
                                                    nullptr);
    g.x = A; g.rexp = c->doz_pat; g.out = y; g.near = c->doz_ws; g.nsplit = nsplit; g.facy = facy;
    g.nredo = e.nredo; g.redo = e.redo;
    k_split64<OZ_RECEIVE><<<ncb * c->noz_tiles, OZ_THREADS, OZ_SMEM, s>>>(g);
    k_redo_receive_near<<<OZ_REDO_CTAS * c->nsm, OZ_REDO_T, 0, s>>>(g.K2, c->N, nrhs, ld, e.nredo, e.redo, g.perm,
                                                              c->dbox_of_sorted, g.R, A, g.ia, g.ja, c->dZd, x, facy, y);
    return cuda_ok(c, cudaGetLastError(), "near + receive (split)") ? MLF_OK : MLF_E_CUDA;
}

// Dense operator: y = Z x for blocks of columns.  The row exponents are bounds by
// blocks of 32 unknowns, so that a product reads the matrix once.  FP64 FMAs, four
// columns a pass, against here: 6750 unknowns x 3: 1399, 470 us; x 24: 7678, 1297;
// 3000 x 2: 339, 120; 1920 x 4: 131, 59; 1080 x 6: 86, 39.  At most OZ_DENSE_COLS
// columns at a time, so that the workspace is made with the context and products
// of any number of columns allocate nothing (the first one may be captured).
int dense64_setup(Ctx* c) {
    const int N = c->N, nblk = (N + 31) / 32;
    CK(cudaDeviceGetAttribute(&c->nsm, cudaDevAttrMultiProcessorCount, c->dev));
    // a limit of the kernel, the same for every context
    CK(cudaFuncSetAttribute(k_split64<OZ_DENSE>, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM));
    c->noz_tiles = (N + OZ_R - 1) / OZ_R;
    CK(cudaMalloc(&c->doz_pat, (size_t)N * nblk * sizeof(short)));
    k_dense_block_exp<<<(N + 7) / 8, 256, 0, c->stream>>>(N, nblk, c->dZdense, reinterpret_cast<short*>(c->doz_pat));
    CK(cudaGetLastError());
    return oz_workspace(c, OZ_DENSE_COLS, 2 * (size_t)N + 1 + nblk, 1 + (size_t)N);
}

static void dense64_columns(Ctx* c, const double2* x, double2* y, int nrhs, int ld, cudaStream_t s) {
    const int N = c->N, nblk = (N + 31) / 32, nsplit = near64_split(c, nrhs);
    int *sexp = c->doz_exp, *rexp = sexp + N, *nredo = rexp + N, *bmax = nredo + 1, *cexp = bmax + nblk;
    unsigned* redo = reinterpret_cast<unsigned*>(cexp + nrhs);
    k_row_exp<<<(N + 255) / 256, 256, 0, s>>>(N, nrhs, ld, x, sexp, nredo, cexp);
    k_dense_col_exp<<<std::min((nblk + 7) / 8, 256), 256, 0, s>>>(N, nrhs, ld, nblk, x, sexp, bmax, cexp);
    k_dense_row_exp<<<(N + 7) / 8, 256, 0, s>>>(N, nblk, reinterpret_cast<const short*>(c->doz_pat), bmax, rexp);
    OzArgs g{};
    g.N = N; g.nrhs = nrhs; g.ld = ld; g.K2 = 1;
    g.R = c->dZdense; g.x = x;
    g.sexp = sexp; g.rexp = rexp; g.cexp = cexp;
    g.out = c->doz_ws; g.cov = oz_covers(c);
    k_split64<OZ_DENSE><<<dim3((unsigned)c->noz_tiles * ((nrhs + OZ_C - 1) / OZ_C), nsplit), OZ_THREADS, OZ_SMEM, s>>>(g);
    k_sum_parts<<<dim3((N + 255) / 256, nrhs), 256, 0, s>>>(N, nrhs, ld, nsplit, c->doz_ws, g.cov, y, nredo, redo);
    k_redo_dense<<<OZ_REDO_CTAS * c->nsm, OZ_REDO_T, 0, s>>>(N, ld, nredo, redo, c->dZdense, x, y);
}

int dense64_matvec(Ctx* c, const double2* x, double2* y, int nrhs, int ld, cudaStream_t s) {
    const int groups = (nrhs + OZ_DENSE_COLS - 1) / OZ_DENSE_COLS;
    const int per = ((nrhs + groups - 1) / groups + OZ_C - 1) / OZ_C * OZ_C;   // whole blocks of 12
    for (int c0 = 0; c0 < nrhs; c0 += per)
        dense64_columns(c, x + (size_t)c0 * ld, y + (size_t)c0 * ld, std::min(per, nrhs - c0), ld, s);
    return cuda_ok(c, cudaGetLastError(), "dense matvec (split)") ? MLF_OK : MLF_E_CUDA;
}

}  // namespace mlf
