// Box-block GEMMs of the FP32 operator on the fifth-generation tensor cores
// (block engine 4): the near field, the leaf aggregation and the leaf receive
// (and the near-pattern preconditioner), as tcgen05.mma with TMEM
// accumulators, operands staged into shared memory by TMA
// (cp.async.bulk.tensor) through tensor maps over this GPU's own memory,
// hi and lo parts of each factor for FP32 accuracy.
//
// The near matrix (llenarZesparcida, modMLFMA.f90:1594-1634) is a union of
// dense box-pair blocks Z_ij (bases of leaf box i x bases of near box j).  For
// a block of right-hand sides, leaf box i needs Y_i = sum_j Z_ij X_j.  Here it
// is computed transposed, as a real GEMM whose M side is the right-hand sides
// (A the right-hand sides, B the box's rows, both with the contraction along rows).
// Near field and aggregation (FP16 operands) take two real products per tile,
//   A row 2c = Xr(:, c), row 2c+1 = Xi(:, c);   B row p = [ Zr(p, :) | Zi(p, :) ]
//   D1 = A Zr^T, D2 = A Zi^T;   Re Y = D1(2c) - D2(2c+1), Im Y = D1(2c+1) + D2(2c)
// combined in the epilogue; the receive (TF32 operands) one on twice the length,
//   A row 2c   = [ Xr(t,c), -Xi(t,c) ]_t   -> D row 2c   = Re Y(:, c)
//   A row 2c+1 = [ Xi(t,c),  Xr(t,c) ]_t   -> D row 2c+1 = Im Y(:, c)
//   B row p    = [ Zr(p,t),  Zi(p,t) ]_t
// The first form reads half the A bytes and accumulates over half the length
// (7680 RWG: 3.7e-6 from FP64 instead of 6.2e-6); its pair of accumulators fits
// TMEM twice only up to 128 rows.  Either way M = 128 covers 64 right-hand sides
// exactly and N = the box's bases
// (padded to 16), with no padding of the rows to 128.  The leaf aggregation
// (llenar_campoCyB, modMLFMA.f90:1805-1811: C_b = R_b^T x_b) and receive
// (MatxVec_MLFMA, modMLFMA.f90:1915-1924: y_b = j facy conj(R_b) A_b) are the
// same GEMM with the patterns R in place of Z.
//
// Layouts in HBM (built once per context; the X operand once per call):
//   Z operand: per block e = (i, j) and chunk kc of 32 columns t, the n_i rows p
//     of [32 re | 32 im] (zero past n_j) in scaled FP16, rows of all blocks and
//     chunks stacked: one 2-D tensor map of 128-byte rows, boxes of 32 rows; hi
//     and lo copies.
//   X operand: per column tile of 64 right-hand sides, per box j and chunk kc, 128
//     rows of 32 FP16, hi and lo; a tensor map of 64-byte rows, boxes of 128 rows.
//   Aggregation / receive operands: R^T as the Z operand, conj R as rows of 16
//     (re, im) pairs in TF32 (tc_leaf_setup); the receive's right-hand side
//     operand is the leaf A field itself, read raw.
// Each TMA box of an operand is written with 128-byte (X: 64-byte) swizzling, the
// canonical K-major SWIZZLE_128B / 64B layouts tcgen05.mma reads (8-row atoms of
// 1024 / 512 bytes).
//
// A persistent CTA (8 warps, the receive's 10) per SM walks its share of the work
// (tiles of at most 160 rows, 64 columns, cut into parts where shares meet, the
// parts' sums added by k_tc_sum).  Thread 0 issues the TMA loads of a ring of
// three to five stages; thread 32 issues the MMAs: per chunk 4 K-steps x 3 products
// (A_lo B_hi, A_hi B_lo, A_hi B_hi) into 128 x N FP32 accumulators in TMEM, and
// tcgen05.commit frees a stage once its MMAs are done.  Warps 4-7 read their
// 32 TMEM lanes each (tcgen05.ld), pair the real and imaginary rows by shuffles and
// write the output, while the next item accumulates into the other TMEM buffer.
//
// Every wait on an mbarrier is bounded; on a timeout the CTA records an error
// flag, lets its loads in flight land, frees its TMEM and skips the output.
// The host checks the flag after the solve (tc_check).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "mlf_cvt.cuh"
#include "mlf_internal.h"
#include "mlf_tcgen05.h"

namespace mlf {

#define CK(call)                                             \
    do {                                                     \
        if (!cuda_ok(c, (call), #call)) return MLF_E_CUDA;   \
    } while (0)

constexpr int TC_ROWS = 160;                 // bases of box i per tile (MMA N <= 160 here)
constexpr int TC_KCH = 16;                   // complex contraction values per 128-byte TF32 row (receive)
constexpr int TC_KCH_H = 32;                 // complex contraction values per 128-byte FP16 row (near, aggregation)
constexpr int TC_COLS = 64;                  // right-hand sides per column tile (MMA M = 128)
constexpr int TC_ZBOX = 32;                  // rows per TMA box of the B operands
constexpr int TC_ABYTES = 128 * 128;         // an A tile of 128-byte rows
// The ring of a mode (TCM_*): for tiles of up to 160 rows four stages of 56 KB
// (the receive, whose A tiles are expanded, three of 72), where no tile has more
// than 96 five of 40 KB (four of 56)
template <int MODE, bool LOW> struct TcRing {
    static constexpr bool RAW = MODE == 2;
    static constexpr int ST = (RAW ? 3 : 4) + LOW;
    static constexpr int ROWS = LOW ? 96 : TC_ROWS;
    static constexpr int ABYTES = RAW ? TC_ABYTES : TC_ABYTES / 2;   // one A tile
    static constexpr int BBYTES = ROWS * 128;                       // one B tile at most
    static constexpr int STAGE = 2 * ABYTES + 2 * BBYTES;
    static constexpr size_t SMEM = (size_t)ST * STAGE + 1024;       // + alignment of the ring
};
constexpr int TC_PARTS = 15;                 // parts of a tile at most (about)
constexpr uint32_t TC_TMEM_COLS = 256;
constexpr uint32_t TC_SPIN = 1u << 20;       // mbarrier polls before a wait gives up

// An operand in rows of 128 bytes: 16 complex values as TF32 (re, im) pairs, or 32
// as FP16, real parts before imaginary ones, scaled by a power of two per output
// row (rinv holds the inverse scales); hi and lo parts.
struct TcOperand {
    void* hi = nullptr;
    void* lo = nullptr;
    float* rinv = nullptr;
    CUtensorMap mhi, mlo;
};

// A GEMM's work in shares for the persistent CTAs: items (tile, run of its chunks)
struct TcSlots {
    int n = 0;                      // shares
    int* ptr = nullptr;             // share -> its items
    int4* item = nullptr;           // (box, first row, rows, part of the tile)
    int2* ch = nullptr;             // first chunk, chunks
    int parts = 0;                  // parts of a tile at most
    unsigned char* np = nullptr;    // per box-sorted basis: parts of its tile
};

struct TcState {
    int nchunk = 0;                 // chunks of 32 bases over all boxes
    long long zrows = 0;            // rows of the Z-operand layout
    int nsm = 0;                    // SMs: CTAs of the persistent GEMM
    std::vector<int4> tiles;        // (box, first row, rows, -)
    int maxrows = 0;                // rows of the largest
    TcSlots near, recv, agg;
    int2* dlist = nullptr;          // near chunks of each box in order: (chunk of the X operand, Z-operand row)
    float2* dws = nullptr;          // parts' sums [part][box-sorted basis][column], the near field's, then the receive's
    size_t ws_cap = 0;
    int* dzrow = nullptr;           // per block entry e: first Z-operand row (chunk 0)
    int* dcbase = nullptr;          // per box: its first chunk
    int2* dchunk = nullptr;         // per chunk: (first box-sorted position, bases in it)
    int* derr = nullptr;            // set by a CTA whose wait gave up
    unsigned* drowmax = nullptr;    // scratch: per box-sorted basis, the largest magnitude of its near row
    TcOperand Z;
    TcOperand M;                    // the neighbourhood-inverse preconditioner on the near pattern (hi null: not built)
    void *xhi = nullptr, *xlo = nullptr;   // X operand (FP16)
    unsigned* dcmax = nullptr;      // per column: largest magnitude
    float* dcinv = nullptr;         // per column: inverse of its power-of-two scale
    long long xrows_cap = 0;
    int cols_cap = 0;
    CUtensorMap mxhi, mxlo;
    // leaf aggregation and receive (built from the FP32 patterns R on first use)
    const float2* Rsrc = nullptr;   // the patterns the operands below hold
    int K2 = 0;                     // 2K directions of the leaf level
    int arows = 0;                  // rows of the largest aggregation tile
    int* dabase = nullptr;          // per box: first row of the aggregation operand
    int* drbase = nullptr;          // per box: first row of the receive operand
    TcOperand RA;                   // R^T per box and chunk of 32 bases: 2K rows of 32 FP16 (re, im)
    TcOperand RR;                   // conj R per box and chunk of 16 directions: n_b rows of 16 TF32 (re, im)
};

// ---------------------------------------------------------------------------
// operand layouts
// ---------------------------------------------------------------------------

// FP16 scaling: the power of two that takes the largest magnitude m of a row
// (or column) into [2^14, 2^15).  Applying and undoing it is exact; the hi
// part then stays inside the FP16 range and the lo part (2^-11 of it) in its
// normal range for every entry within 2^-14 of m, so the hi/lo split keeps
// the same 22 bits as the TF32 split.
__device__ __forceinline__ int h_scale_exp(float m) {
    if (!(m > 0.f) || !isfinite(m)) return 0;
    int ex;
    frexpf(m, &ex);   // m = f 2^ex, f in [0.5, 1)
    return 15 - ex;
}

__device__ __forceinline__ __half2 h_hi(float a, float b) { return __floats2half2_rn(a, b); }
__device__ __forceinline__ __half2 h_lo(float a, float b, __half2 hi) {
    const float2 h = __half22float2(hi);
    return __floats2half2_rn(a - h.x, b - h.y);
}

// rowmax[i0 + p] = max over the block's row p of |re|, |im| (atomic over the
// near boxes of box i); one CTA per block entry, a thread per row
__global__ void k_blk_rowmax(const int* __restrict__ entry_box, const int* __restrict__ nbox_list,
                             const long long* __restrict__ blk_off, const int* __restrict__ box_ptr,
                             const float2* __restrict__ blk, unsigned* __restrict__ rowmax) {
    const int e = blockIdx.x;
    const int i = entry_box[e], j = nbox_list[e];
    const int i0 = box_ptr[i], ni = box_ptr[i + 1] - i0, nj = box_ptr[j + 1] - box_ptr[j];
    const float2* src = blk + blk_off[e];
    for (int p = threadIdx.x; p < ni; p += blockDim.x) {
        float m = 0.f;
        for (int t = 0; t < nj; ++t) {
            const float2 v = src[(size_t)t * ni + p];
            m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
        }
        atomicMax(rowmax + i0 + p, __float_as_uint(m));
    }
}

__global__ void k_rinv(int n, const unsigned* __restrict__ rowmax, float* __restrict__ rinv) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) rinv[k] = ldexpf(1.f, -h_scale_exp(__uint_as_float(rowmax[k])));
}

// Values v, w of places 2u, 2u + 1, scaled by 2^ex, to a row's [32 re][32 im], hi
// and lo; o = the row's first pair + u
__device__ __forceinline__ void put_planar(__half2* __restrict__ hi, __half2* __restrict__ lo, size_t o, float2 v,
                                           float2 w, int ex) {
    const float a = ldexpf(v.x, ex), b = ldexpf(w.x, ex), c = ldexpf(v.y, ex), d = ldexpf(w.y, ex);
    const __half2 r = h_hi(a, b), i = h_hi(c, d);
    hi[o] = r;
    hi[o + TC_KCH_H / 2] = i;
    lo[o] = h_lo(a, b, r);
    lo[o + TC_KCH_H / 2] = h_lo(c, d, i);
}

// Z operand of block entry e (one CTA each) from the box-pair blocks (column-
// major n_i x n_j at blk_off[e]): row zrow[e] + kc n_i + p holds
// s_p Z(p, 32 kc + u), u = 0..31, as FP16 (re, im) pairs, hi and lo, with
// s_p the power-of-two scale of target basis p's near row.
__global__ void k_tc_fill_zh(const int* __restrict__ entry_box, const int* __restrict__ nbox_list,
                             const long long* __restrict__ blk_off, const int* __restrict__ box_ptr,
                             const int* __restrict__ zrow, const float2* __restrict__ blk,
                             const unsigned* __restrict__ rowmax, __half2* __restrict__ zhi,
                             __half2* __restrict__ zlo) {
    const int e = blockIdx.x;
    const int i = entry_box[e], j = nbox_list[e];
    const int i0 = box_ptr[i], ni = box_ptr[i + 1] - i0, nj = box_ptr[j + 1] - box_ptr[j];
    const int nkc = (nj + TC_KCH_H - 1) / TC_KCH_H;
    const float2* src = blk + blk_off[e];
    const size_t base = (size_t)zrow[e] * TC_KCH_H;
    for (int q = threadIdx.x; q < nkc * ni * (TC_KCH_H / 2); q += blockDim.x) {
        const int u = q % (TC_KCH_H / 2), rp = q / (TC_KCH_H / 2);     // rp = kc n_i + p
        const int kc = rp / ni, p = rp - kc * ni;
        const int t = kc * TC_KCH_H + 2 * u;
        const float2 v = t < nj ? src[(size_t)t * ni + p] : make_float2(0.f, 0.f);
        const float2 w = t + 1 < nj ? src[(size_t)(t + 1) * ni + p] : make_float2(0.f, 0.f);
        put_planar(zhi, zlo, base + (size_t)rp * TC_KCH_H + u, v, w, h_scale_exp(__uint_as_float(rowmax[i0 + p])));
    }
}

// cmax[col] = max over column col of xs (box-sorted rows, row-major N x nrhs)
// of |re|, |im|; grid (N / 64, nrhs / 64), 64 columns x 4 row groups per CTA.
// A thread's rows are a chain of loads: 16 of them, eight in flight, where 64 on
// a quarter of the CTAs took 10.2 us for 15360 x 32.
__global__ void __launch_bounds__(256) k_tc_colmax(int N, int nrhs, const float2* __restrict__ xs,
                                                   unsigned* __restrict__ cmax) {
    __shared__ float red[4][TC_COLS];
    const int tx = threadIdx.x & (TC_COLS - 1), ty = threadIdx.x / TC_COLS;
    const int col = blockIdx.y * TC_COLS + tx;
    const int r0 = blockIdx.x * 64 + ty * 16, r1 = min(r0 + 16, N);
    float m = 0.f;
    if (col < nrhs)
#pragma unroll 8
        for (int r = r0; r < r1; ++r) {
            const float2 v = xs[(size_t)r * nrhs + col];
            m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
        }
    red[ty][tx] = m;
    __syncthreads();
    if (ty == 0 && col < nrhs)
        atomicMax(cmax + col, __float_as_uint(fmaxf(fmaxf(red[0][tx], red[1][tx]), fmaxf(red[2][tx], red[3][tx]))));
}

// X operand of one (column tile, chunk of 32 bases) per CTA from xs: rows 2c
// and 2c+1 of the chunk's 128 as in the header, scaled by column c's power of
// two, FP16 hi and lo; cinv receives the inverse scales.
__global__ void __launch_bounds__(256) k_tc_pack_xh(int nchunk, int nrhs, const int2* __restrict__ chunk,
                                                    const float2* __restrict__ xs, const unsigned* __restrict__ cmax,
                                                    __half2* __restrict__ xhi, __half2* __restrict__ xlo,
                                                    float* __restrict__ cinv) {
    __shared__ float2 xsm[TC_KCH_H][TC_COLS + 1];
    __shared__ int sexp[TC_COLS];
    const int ch = blockIdx.x, ct = blockIdx.y;
    const int2 cd = chunk[ch];
    if (threadIdx.x < TC_COLS) {
        const int col = ct * TC_COLS + threadIdx.x;
        const int ex = col < nrhs ? h_scale_exp(__uint_as_float(cmax[col])) : 0;
        sexp[threadIdx.x] = ex;
        if (ch == 0 && col < nrhs) cinv[col] = ldexpf(1.f, -ex);
    }
    for (int q = threadIdx.x; q < TC_KCH_H * TC_COLS; q += blockDim.x) {
        const int u = q / TC_COLS, cl = q - u * TC_COLS, col = ct * TC_COLS + cl;
        xsm[u][cl] = (u < cd.y && col < nrhs) ? xs[(size_t)(cd.x + u) * nrhs + col] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    const size_t base = ((size_t)ct * nchunk + ch) * 128 * (TC_KCH_H / 2);
    for (int q = threadIdx.x; q < 128 * (TC_KCH_H / 2); q += blockDim.x) {
        const int row = q / (TC_KCH_H / 2), u = 2 * (q - row * (TC_KCH_H / 2));
        const float2 v = xsm[u][row >> 1], w = xsm[u + 1][row >> 1];
        const int ex = sexp[row >> 1];
        const float a = ldexpf((row & 1) ? v.y : v.x, ex), b = ldexpf((row & 1) ? w.y : w.x, ex);
        const __half2 h = h_hi(a, b);
        xhi[base + q] = h;
        xlo[base + q] = h_lo(a, b, h);
    }
}

// Aggregation operand of box b (one CTA per box): row abase[b] + kc 2K + q
// holds s_bq R(32 kc + u, q) for u = 0..31 (zero past the box's bases) as FP16
// hi and lo, s_bq the power-of-two scale of direction q over the box's bases;
// rinv[b 2K + q] = 1 / s_bq.
__global__ void k_tc_fill_rah(int K2, const int* __restrict__ box_ptr, const int* __restrict__ abase,
                              const float2* __restrict__ R, __half2* __restrict__ hi, __half2* __restrict__ lo,
                              float* __restrict__ rinv) {
    const int b = blockIdx.x;
    const int j0 = box_ptr[b], n = box_ptr[b + 1] - j0;
    const int nkc = (n + TC_KCH_H - 1) / TC_KCH_H;
    const size_t base = (size_t)abase[b] * TC_KCH_H;
    for (int q = threadIdx.x; q < K2; q += blockDim.x) {
        float m = 0.f;
        for (int t = 0; t < n; ++t) {
            const float2 v = R[(size_t)(j0 + t) * K2 + q];
            m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
        }
        const int ex = h_scale_exp(m);
        rinv[(size_t)b * K2 + q] = ldexpf(1.f, -ex);
        for (int kc = 0; kc < nkc; ++kc)
            for (int u = 0; u < TC_KCH_H / 2; ++u) {
                const int t = kc * TC_KCH_H + 2 * u;
                const float2 v = t < n ? R[(size_t)(j0 + t) * K2 + q] : make_float2(0.f, 0.f);
                const float2 w = t + 1 < n ? R[(size_t)(j0 + t + 1) * K2 + q] : make_float2(0.f, 0.f);
                put_planar(hi, lo, base + ((size_t)kc * K2 + q) * TC_KCH_H + u, v, w, ex);
            }
    }
}

// Receive operand of box b: row rbase[b] + kc n_b + p holds conj R(p, 16 kc + u)
// for u = 0..15 (zero past the 2K directions).
__global__ void k_tc_fill_rr(int K2, const int* __restrict__ box_ptr, const int* __restrict__ rbase,
                             const float2* __restrict__ R, float* __restrict__ hi, float* __restrict__ lo) {
    const int b = blockIdx.x;
    const int j0 = box_ptr[b], n = box_ptr[b + 1] - j0;
    const int nqc = (K2 + TC_KCH - 1) / TC_KCH;
    const size_t base = (size_t)rbase[b] * 32;
    for (long long e = threadIdx.x; e < (long long)n * nqc * TC_KCH; e += blockDim.x) {
        const int qq = (int)(e % (nqc * TC_KCH));      // 16 kc + u
        const int p = (int)(e / (nqc * TC_KCH));
        const int kc = qq / TC_KCH, u = qq - kc * TC_KCH;
        float2 v = qq < K2 ? R[(size_t)(j0 + p) * K2 + qq] : make_float2(0.f, 0.f);
        v.y = -v.y;
        const float hr = tc::tf32_rna(v.x), hi_ = tc::tf32_rna(v.y);
        const size_t o = base + ((size_t)kc * n + p) * 32 + 2 * u;
        *reinterpret_cast<float2*>(hi + o) = make_float2(hr, hi_);
        *reinterpret_cast<float2*>(lo + o) = make_float2(tc::tf32_rna(v.x - hr), tc::tf32_rna(v.y - hi_));
    }
}

// ---------------------------------------------------------------------------
// the GEMM
// ---------------------------------------------------------------------------

// What one launch computes (B the operand streamed by TMA, X the right-hand
// side operand, item = (box i, first row r0, rows, part)):
//   TCM_NEAR      part of Z X (or M X, M on the near pattern) over the near boxes j
//                 of box i, to ws
//   TCM_AGG       C(q, col, i) = sum_t R(t, q) x(t, col), t over box i's bases,
//                 q = r0 .. r0 + rows - 1 of the 2K directions
//   TCM_RECV      part of j facy sum_q conj R(basis, q) A(q, col, i), to ws
// The aggregation takes the near field's packed X operand (the box's own
// chunks); the receive stages raw rows of the A field (64 columns x 16
// directions, 128-byte swizzled) by TMA and warps 2, 3, 8, 9 expand them in shared memory
// into the [re, -im] / [im, re] row pairs, split into TF32 hi and lo.
//
// Persistent: one CTA per SM takes the shares (tc_slots) and column tiles q =
// blockIdx.x + k gridDim.x, the column tiles of a share on neighbouring CTAs, which
// read the same B rows.  Warp roles: warp 0 lane 0 issues the TMA loads, warp 1
// lane 0 the MMAs, warps 2, 3, 8, 9 expand the receive's raw rows, warps 4-7 read
// the accumulators out (warp 4 + w owns TMEM lanes 32 w .. 32 w + 31).  Two
// TMEM accumulators of 256 columns alternate between items, so the loads and
// MMAs of the next item run under the epilogue of the previous one; the
// shared-memory ring and its barrier phases run on across items.
enum : int { TCM_NEAR = 0, TCM_AGG = 1, TCM_RECV = 2 };

struct TcArgs {
    int nslots, nct;         // shares of the work, column tiles of 64
    int nbuf;                // accumulators (pairs of them) in TMEM
    const int* slot;         // TcSlots ptr, item, ch
    const int4* item;
    const int2* ch;
    const int* box_ptr;
    const int2* list;        // near: chunks of the boxes' near lists
    const int* zrow;         // aggregation, receive: per box -- first B row
    const int* cbase;        // aggregation: per box, its first chunk of the X operand
    int nchunk, nrhs, K2, N;
    float facy;
    const float* rinv;       // FP16 modes: per output row (near: box-sorted basis; aggregation: box x 2K), 1 / scale
    const float* cinv;       // FP16 modes: per column, 1 / scale
    float2* C;               // aggregation
    float2* ws;              // near, receive: parts' sums, for k_tc_sum
    int* err;
};

// Operands of the near field, its preconditioner and the aggregation are FP16
// (kind::f16, 32 complex values per 128-byte row); the receive's are TF32
// (kind::tf32, 16 per row).  Either way a K step is 32 bytes of the row.
template <int MODE>
struct TcFmt {
    static constexpr bool H = MODE != TCM_RECV;
    static constexpr uint32_t FMT = H ? tc::FMT_F16 : tc::FMT_TF32;
    static constexpr int KCH = H ? TC_KCH_H : TC_KCH;
};

template <int MODE>
constexpr int TC_THREADS = MODE == TCM_RECV ? 320 : 256;

template <int MODE, bool LOW>
__global__ void __launch_bounds__(TC_THREADS<MODE>, 1)
    k_tc_gemm(const __grid_constant__ CUtensorMap mbhi, const __grid_constant__ CUtensorMap mblo,
              const __grid_constant__ CUtensorMap mxhi, const __grid_constant__ CUtensorMap mxlo, const TcArgs a) {
    constexpr bool NEAR = MODE == TCM_NEAR;
    constexpr bool RAW = MODE == TCM_RECV;
    using Ring = TcRing<MODE, LOW>;
    constexpr int ST = Ring::ST, STAGE = Ring::STAGE, ABYTES = Ring::ABYTES, BBYTES = Ring::BBYTES;
    constexpr uint32_t RAW_BYTES = TC_COLS * 128;   // 64 field rows of 16 complex values
    extern __shared__ unsigned char tc_raw[];
    __shared__ __align__(8) uint64_t full[ST], empty[ST], conv[ST], accf[2], acce[2], done;
    __shared__ uint32_t tmem_base;
    __shared__ int fail_s, cvok_s, issued_s, consumed_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t raw = tc::smem_u32(tc_raw);
    unsigned char* ring = tc_raw + (((raw + 1023u) & ~1023u) - raw);   // 1024-aligned swizzle atoms
    const int nwork = a.nslots * a.nct;
    const uint32_t nbuf = (uint32_t)a.nbuf, dim = nbuf == 2 ? TC_TMEM_COLS / 2 : TC_TMEM_COLS;   // second accumulator of a pair
    volatile int* vfail = &fail_s;
    if (tid == 0) {
        for (int s = 0; s < ST; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
            tc::mbar_init(&conv[s], 128);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accf[b], 1);
            tc::mbar_init(&acce[b], 128);
        }
        tc::mbar_init(&done, 1);
        tc::fence_barrier_init();
        // once any CTA has given up a wait, the rest skip their work (the call fails anyway)
        fail_s = *reinterpret_cast<volatile int*>(a.err) ? 1 : 0;
        issued_s = consumed_s = 0;
    }
    if (warp == 0) {
        tc::tmem_alloc(&tmem_base, 2 * TC_TMEM_COLS);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem = tmem_base;
    const bool skip_all = fail_s != 0;

    if (warp == 0) {
        if (lane == 0 && !skip_all) {
            // producer: TMA loads of chunk g into stage g % STAGES once that stage's MMAs are done
            tc::tma_prefetch_desc(&mbhi);
            tc::tma_prefetch_desc(&mblo);
            tc::tma_prefetch_desc(&mxhi);
            if (!RAW) tc::tma_prefetch_desc(&mxlo);
            // the B operands stream through once (evicted first from L2); the X
            // operand, read again by the CTAs of every target box near its source
            // box, keeps the normal policy, as does everything after this kernel
            const uint64_t pol_b = tc::l2_evict_first();
            uint32_t g = 0;
            bool ok = true;
            for (int q = blockIdx.x; q < nwork && ok; q += gridDim.x) {
            const int sl = q / a.nct, ct = q - sl * a.nct, t1 = a.slot[sl + 1];
            for (int it = a.slot[sl]; it < t1 && ok; ++it) {
                const int4 tl = a.item[it];
                const int2 ch = a.ch[it];
                const int i = tl.x, r0 = tl.y, nrow = tl.z, nch = ch.y;
                const int ni = a.box_ptr[i + 1] - a.box_ptr[i];
                const int nB = (nrow + TC_ZBOX - 1) / TC_ZBOX * TC_ZBOX;          // B rows staged
                const uint32_t bytes = (RAW ? RAW_BYTES : 2u * ABYTES) + 2u * (uint32_t)nB * 128u;
                int2 next = NEAR && nch ? a.list[ch.x] : make_int2(0, 0);   // a chunk ahead of its use
                for (int cI = 0; cI < nch; ++cI, ++g) {
                    const int s = g % ST;
                    if ((g >= ST && !tc::mbar_wait(&empty[s], ((g / ST) - 1) & 1, TC_SPIN)) || *vfail) {
                        ok = false;   // the consumers then give up on this stage's full barrier too
                        break;
                    }
                    unsigned char* st = ring + (size_t)s * STAGE;
                    tc::mbar_arrive_expect_tx(&full[s], bytes);
                    int zr;
                    if (NEAR) {
                        const int xr = (ct * a.nchunk + next.x) * 128;
                        zr = next.y + r0;
                        tc::tma_load_2d(st, &mxhi, 0, xr, &full[s]);
                        tc::tma_load_2d(st + ABYTES, &mxlo, 0, xr, &full[s]);
                        if (cI + 1 < nch) next = a.list[ch.x + cI + 1];
                    } else if (MODE == TCM_AGG) {
                        const int xr = (ct * a.nchunk + a.cbase[i] + cI) * 128;
                        tc::tma_load_2d(st, &mxhi, 0, xr, &full[s]);
                        tc::tma_load_2d(st + ABYTES, &mxlo, 0, xr, &full[s]);
                        zr = a.zrow[i] + cI * a.K2 + r0;
                    } else {
                        // raw field rows (box i, columns of this tile) into the lo tile's first 8 KB
                        tc::tma_load_2d_hint(st + ABYTES, &mxhi, 2 * TC_KCH * (ch.x + cI), i * a.nrhs + ct * TC_COLS,
                                             &full[s], pol_b);
                        zr = a.zrow[i] + (ch.x + cI) * ni + r0;
                    }
                    // the aggregation's and receive's pattern operands are read by the
                    // tiles of one box (and the column tiles) only: streamed too
                    for (int qq = 0; qq < nB; qq += TC_ZBOX) {
                        tc::tma_load_2d_hint(st + 2 * ABYTES + qq * 128, &mbhi, 0, zr + qq, &full[s], pol_b);
                        tc::tma_load_2d_hint(st + 2 * ABYTES + BBYTES + qq * 128, &mblo, 0, zr + qq, &full[s], pol_b);
                    }
                }
            }
            }
            issued_s = (int)g;
            if (!ok) *vfail = 1;
        }
    } else if (warp == 1) {
        if (lane == 0 && !skip_all) {
            // MMA issuer: per chunk 4 K steps x 3 products into the item's TMEM accumulator
            uint32_t g = 0, na = 0;
            bool ok = true;
            for (int q = blockIdx.x; q < nwork && ok; q += gridDim.x) {
            const int sl = q / a.nct, t1 = a.slot[sl + 1];
            for (int it = a.slot[sl]; it < t1; ++it) {
                const int nch = a.ch[it].y;
                if (nch == 0) continue;
                const uint32_t buf = na % nbuf;
                if (na >= nbuf && !tc::mbar_wait(&acce[buf], (na / nbuf - 1) & 1, TC_SPIN)) {
                    ok = false;
                    break;
                }
                tc::tc_fence_after_sync();
                const uint32_t d = tmem + buf * TC_TMEM_COLS;
                const uint32_t idesc = tc::instr_desc_f32acc(TcFmt<MODE>::FMT, 128, (a.item[it].z + 15) / 16 * 16);
                for (int cI = 0; cI < nch; ++cI, ++g) {
                    const int s = g % ST;
                    const uint32_t par = (g / ST) & 1;
                    if (!tc::mbar_wait(&full[s], par, TC_SPIN) || (RAW && !tc::mbar_wait(&conv[s], par, TC_SPIN))) {
                        ok = false;
                        break;
                    }
                    tc::tc_fence_after_sync();
                    const uint32_t st = tc::smem_u32(ring + (size_t)s * STAGE);
                    const uint32_t ahi = st, alo = st + ABYTES, bhi = st + 2 * ABYTES, blo = bhi + BBYTES;
                    if constexpr (RAW) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) {   // K steps of 32 bytes of the 128-byte rows
                            const uint32_t ko = 32u * k;
                            const uint64_t dal = tc::kmajor_sw128_desc(alo + ko), dah = tc::kmajor_sw128_desc(ahi + ko);
                            const uint64_t dbl = tc::kmajor_sw128_desc(blo + ko), dbh = tc::kmajor_sw128_desc(bhi + ko);
                            tc::mma_tf32(d, dal, dbh, idesc, (cI | k) != 0);
                            tc::mma_tf32(d, dah, dbl, idesc, 1);
                            tc::mma_tf32(d, dah, dbh, idesc, 1);
                        }
                    } else {
                        // K steps of 32 bytes of A's 64-byte rows, against Zr and Zi
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t ka = 32u * (k >> 1), kb = ka + 64u * (k & 1), dd = d + (k & 1 ? dim : 0u);
                            const uint64_t dal = tc::kmajor_sw64_desc(alo + ka), dah = tc::kmajor_sw64_desc(ahi + ka);
                            const uint64_t dbl = tc::kmajor_sw128_desc(blo + kb), dbh = tc::kmajor_sw128_desc(bhi + kb);
                            tc::mma_f16(dd, dal, dbh, idesc, (cI | (k >> 1)) != 0);
                            tc::mma_f16(dd, dah, dbl, idesc, 1);
                            tc::mma_f16(dd, dah, dbh, idesc, 1);
                        }
                    }
                    tc::mma_commit(&empty[s]);
                }
                if (!ok) break;
                tc::mma_commit(&accf[buf]);   // the item's accumulator is complete
                ++na;
            }
            }
            if (g > 0) {
                tc::mma_commit(&done);   // every MMA issued above
                if (!tc::mbar_wait(&done, 0, TC_SPIN)) ok = false;
            }
            consumed_s = (int)g;
            if (!ok) *vfail = 1;
        }
    } else if (warp < 4 || warp >= 8) {
        if (RAW && !skip_all) {
            // converters (warps 2, 3, 8, 9): threads cl and 64 + cl expand half of field row
            // cl (column ct 64 + cl) of each chunk each; with one thread a row this was the
            // receive's time (2350 cycles a chunk)
            const int cid = warp < 4 ? tid - 64 : tid - 192, cl = cid & 63, kh = cid >> 6 << 2;
            uint32_t g = 0;
            bool go = true;
            for (int q = blockIdx.x; q < nwork && go; q += gridDim.x) {
            const int sl = q / a.nct, t1 = a.slot[sl + 1];
            for (int it = a.slot[sl]; it < t1 && go; ++it) {
                const int nch = a.ch[it].y;
                for (int cI = 0; cI < nch; ++cI, ++g) {
                    const int s = g % ST;
                    const uint32_t par = (g / ST) & 1;
                    if (cid == 0) cvok_s = (!*vfail && tc::mbar_wait(&full[s], par, TC_SPIN)) ? 1 : 0;
                    tc::named_bar_sync(1, 128);
                    if (!cvok_s) {   // the same decision in all 128 threads
                        go = false;
                        break;
                    }
                    tc::mbar_wait(&full[s], par, TC_SPIN);   // complete already: acquires the landed bytes
                    unsigned char* st = ring + (size_t)s * STAGE;
                    // the raw rows arrive 128-byte swizzled: chunk k of row cl sits at
                    // k ^ (cl & 7), so the 8 lanes of a shared-memory wavefront read 8
                    // different bank groups
                    float4 v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        v[k] = *reinterpret_cast<const float4*>(st + ABYTES + tc::sw128_offset(cl, kh + k));
                    tc::named_bar_sync(1, 128);   // every raw row is read before the lo tile overwrites them
                    // rows 2cl and 2cl+1 place chunk k at k ^ (2cl & 7) (resp. +1): lanes
                    // with cl & 4 take the chunks in the order k ^ 1 so that the 8 lanes
                    // of a wavefront again store to 8 different bank groups
                    const int flip = (cl >> 2) & 1;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {   // 16-byte chunk k: complex values 2k, 2k+1
                        const int k = kh + (kk ^ flip);
                        const float4 w = flip ? v[kk ^ 1] : v[kk];
                        // row 2cl: (re, -im) pairs; row 2cl+1: (im, re) -- the same values, so
                        // its hi and lo parts follow from row 2cl's (the rounding is symmetric)
                        const float4 eh = make_float4(tc::tf32_rna(w.x), tc::tf32_rna(-w.y), tc::tf32_rna(w.z),
                                                      tc::tf32_rna(-w.w));
                        const float4 el = make_float4(tc::tf32_rna(w.x - eh.x), tc::tf32_rna(-w.y - eh.y),
                                                      tc::tf32_rna(w.z - eh.z), tc::tf32_rna(-w.w - eh.w));
                        const float4 oh = make_float4(-eh.y, eh.x, -eh.w, eh.z);
                        const float4 ol = make_float4(-el.y, el.x, -el.w, el.z);
                        const uint32_t oe = tc::sw128_offset(2 * cl, k), oo = tc::sw128_offset(2 * cl + 1, k);
                        *reinterpret_cast<float4*>(st + oe) = eh;
                        *reinterpret_cast<float4*>(st + oo) = oh;
                        *reinterpret_cast<float4*>(st + ABYTES + oe) = el;
                        *reinterpret_cast<float4*>(st + ABYTES + oo) = ol;
                    }
                    tc::fence_proxy_async_smem();
                    tc::mbar_arrive(&conv[s]);
                }
            }
            }
        }
    } else if (!skip_all) {
        // epilogue: warp 4 + ew reads accumulator rows (TMEM lanes) 32 ew .. 32 ew + 31
        const int ew = warp - 4;
        const int m = 32 * ew + lane;                   // D row = TMEM lane
        uint32_t na = 0;
        bool go = true;
        for (int q = blockIdx.x; q < nwork && go; q += gridDim.x) {
        const int sl = q / a.nct, ct = q - sl * a.nct, t1 = a.slot[sl + 1];
        const int col = ct * TC_COLS + (m >> 1), odd = lane & 1;
        const bool writer = col < a.nrhs;
        const float cs = (TcFmt<MODE>::H && writer) ? a.cinv[col] : 1.f;
        for (int it = a.slot[sl]; it < t1; ++it) {
            const int4 tl = a.item[it];
            const int i = tl.x, r0 = tl.y, nrow = tl.z;
            if (a.ch[it].y == 0) {
                // a box without bases radiates nothing
                if (MODE == TCM_AGG && writer && !odd)
                    for (int p = 0; p < nrow; ++p) a.C[((size_t)i * a.nrhs + col) * a.K2 + r0 + p] = make_float2(0.f, 0.f);
                continue;
            }
            const int i0 = a.box_ptr[i];
            const uint32_t buf = na % nbuf;
            // a warp-uniform decision: tcgen05.ld below is a whole-warp instruction
            const bool got = __all_sync(0xffffffffu, tc::mbar_wait(&accf[buf], (na / nbuf) & 1, TC_SPIN) ? 1 : 0);
            if (!got) {
                *vfail = 1;
                go = false;
                break;
            }
            tc::tc_fence_after_sync();
            const uint32_t d = tmem + buf * TC_TMEM_COLS + ((uint32_t)(32 * ew) << 16);
            for (int n0 = 0; n0 < nrow; n0 += 32) {
                // the rows' inverse scales, one a lane (read row by row between the stores
                // they were 10 000 cycles an item)
                float rl = 1.f;
                if (!RAW && n0 + lane < nrow)
                    rl = __ldg(a.rinv + (MODE == TCM_AGG ? (size_t)i * a.K2 + r0 : (size_t)(i0 + r0)) + n0 + lane);
                float v[32];
                tc::tmem_ld_32x32b_x32(d + (uint32_t)n0, v);
                // lane 2c holds Re and lane 2c + 1 Im of column c; with FP16 operands lane
                // 2c Xr Zr (v) and Xr Zi (w), lane 2c + 1 Xi Zr and Xi Zi.  Half the rows
                // are completed by each of the two.
                float w[32];
                if constexpr (!RAW) tc::tmem_ld_32x32b_x32(d + dim + (uint32_t)n0, w);
                auto value = [&](int e, int o) {   // row e in the even lane, o in the odd lane
                    const float m = odd ? v[o] : v[e], x = __shfl_xor_sync(0xffffffffu, odd ? v[e] : v[o], 1);
                    if constexpr (RAW) return odd ? make_float2(x, m) : make_float2(m, x);
                    const float n = odd ? w[o] : w[e], z = __shfl_xor_sync(0xffffffffu, odd ? w[e] : w[o], 1);
                    return odd ? make_float2(x - n, m + z) : make_float2(m - z, x + n);
                };
                if (MODE == TCM_AGG) {
                    // two rows of four each, 32 bytes of the column's field a pair (8-byte
                    // stores by even lanes were a sector each: 27 000 cycles an item, most
                    // of the kernel)
#pragma unroll
                    for (int u = 0; u < 32; u += 4) {
                        const float2 v0 = value(u, u + 2), v1 = value(u + 1, u + 3);
                        const int p = n0 + u + 2 * odd;
                        const float r0s = __shfl_sync(0xffffffffu, rl, u + 2 * odd) * cs;   // powers of two: exact
                        const float r1s = __shfl_sync(0xffffffffu, rl, u + 2 * odd + 1) * cs;
                        if (writer && p < nrow)   // rows and 2K are even
                            *reinterpret_cast<float4*>(a.C + ((size_t)i * a.nrhs + col) * a.K2 + r0 + p) =
                                make_float4(v0.x * r0s, v0.y * r0s, v1.x * r1s, v1.y * r1s);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < 32; u += 2) {
                        const float2 t = value(u, u + 1);
                        const int p = n0 + u + odd;
                        const float rs = NEAR ? __shfl_sync(0xffffffffu, rl, u + odd) * cs : 1.f;
                        if (writer && p < nrow)
                            a.ws[((size_t)tl.w * a.N + i0 + r0 + p) * a.nrhs + col] =
                                NEAR ? make_float2(t.x * rs, t.y * rs) : make_float2(-(a.facy * t.y), a.facy * t.x);
                    }
                }
            }
            tc::tc_fence_before_sync();
            tc::mbar_arrive(&acce[buf]);   // the MMAs may overwrite this accumulator
            ++na;
        }
        }
    }
    __syncthreads();
    tc::tc_fence_after_sync();
    if (tid == 0 && fail_s) {
        atomicExch(a.err, 1);
        // loads already issued land before the shared memory is given up: at most
        // STAGES chunks beyond the last one the MMA thread consumed
        const uint32_t c0 = (uint32_t)consumed_s, c1 = (uint32_t)issued_s;
        for (uint32_t g = c0; g < c1 && g < c0 + ST; ++g)
            tc::mbar_wait(&full[g % ST], (g / ST) & 1, TC_SPIN);
    }
    tc::tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 2 * TC_TMEM_COLS);
}

// Row n of y = the receive's parts + the near field's, or of out32 = the near
// parts alone: the parts ws[part][pos[n]][col] of each added in order in FP32, as
// they were accumulated, the two sums in FP64.  Tiles of 32 rows x 32 columns
// turned in shared memory, so that both sides move whole sectors.  30720 x 64:
// 70 us with the parts converted and added in FP64 -> 29 us
template <class T2>
__global__ void __launch_bounds__(256) k_tc_sum(int N, int nrhs, int ld, const int* __restrict__ pos,
                                                const unsigned char* __restrict__ npn, const float2* __restrict__ wsn,
                                                const unsigned char* __restrict__ npr, const float2* __restrict__ wsr,
                                                T2* __restrict__ out) {
    constexpr bool Y = sizeof(T2) == sizeof(double2);
    __shared__ float2 t[Y ? 2 : 1][32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, n0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
#pragma unroll
    for (int r = ty; r < 32; r += 8) {
        if (n0 + r >= N || c0 + tx >= nrhs) continue;
        const int p = pos[n0 + r];
        auto sum = [&](int n, const float2* __restrict__ ws) {
            float2 v = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int q = 0; q < n; ++q) {
                const float2 w = ws[((size_t)q * N + p) * nrhs + c0 + tx];
                v.x += w.x;
                v.y += w.y;
            }
            return v;
        };
        t[0][r][tx] = sum(npn[p], wsn);
        if (Y) t[Y][r][tx] = sum(npr[p], wsr);
    }
    __syncthreads();
    if (n0 + tx >= N) return;
    for (int c = ty; c < 32 && c0 + c < nrhs; c += 8) {
        const float2 v = t[0][tx][c], w = t[Y][tx][c];
        T2 o;
        o.x = v.x;
        o.y = v.y;
        if constexpr (Y) {
            o.x = f2d(w.x) + f2d(v.x);
            o.y = f2d(w.y) + f2d(v.y);
        }
        out[(size_t)(c0 + c) * ld + n0 + tx] = o;
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

namespace {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder(Ctx* c) {
    static std::mutex mu;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || !p) {
            c->err = "cuTensorMapEncodeTiled is not available from the driver";
            return nullptr;
        }
        fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
    return fn;
}

// 2-D FP32 tensor map: rows of `inner` floats `row_bytes` apart, boxes of
// box_inner x box_rows, zero fill past the edges
int make_map_2d(Ctx* c, CUtensorMap* m, const void* base, long long inner, long long rows, long long row_bytes,
                int box_inner, int box_rows, CUtensorMapSwizzle swz) {
    auto enc = tensor_map_encoder(c);
    if (!enc) return MLF_E_CUDA;
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)std::max<long long>(rows, 1)};
    const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        c->err = "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")";
        return MLF_E_CUDA;
    }
    return MLF_OK;
}

// operand rows of 32 floats (128 bytes), boxes of box_rows rows, 128-byte swizzle
int make_rows_map(Ctx* c, CUtensorMap* m, const void* base, long long rows, int box_rows) {
    return make_map_2d(c, m, base, 32, rows, 128, 32, box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace

static void tc_slots_free(TcSlots* w) {
    auto F = [](void* p) { if (p) cudaFree(p); };
    F(w->ptr); F(w->item); F(w->ch); F(w->np);
    *w = TcSlots();
}

// The chunks ch[k] (first, number) of the tiles in equal shares, one per SM,
// consecutive in tile order; with split a tile whose chunks fall into several
// shares becomes as many parts (runs of under three chunks join their neighbour).
// Whole tiles per CTA left SMs idle: 184 tiles of the 30720-RWG spheroid's boxes
// need two rounds on 152 SMs, 46 tiles of the 7680-RWG one under a third.  A share
// holds eight chunks or more, a tile about TC_PARTS parts at most.  The FP32
// accumulations are shorter in parts: 7680 RWG are 6.2e-6 from FP64 instead of
// 1.5e-5.  30720 RWG x 64 columns: near field 167 -> 136 us, receive 80 -> 54.
// chunk_cost and item_cost, in rows staged: a line through the CTAs' measured
// times, near field 780 + 4.2 rows cycles a chunk and 10 600 an item, aggregation
// 1500 a chunk and 5100 an item, receive 1420 + 5.1 rows and 670.  By bytes alone
// the last CTA took 25 % (near) to 80 % (aggregation) longer than the mean, now 10 to
// 27 %: near field 136 -> 124 us, aggregation 59 -> 35.
static int tc_slots(Ctx* c, TcSlots* w, const std::vector<int4>& tiles, const std::vector<int2>& ch, bool split,
                    double chunk_cost, double item_cost) {
    tc_slots_free(w);
    auto cost = [&](size_t k) { return chunk_cost + (tiles[k].z + TC_ZBOX - 1) / TC_ZBOX * TC_ZBOX; };   // rows staged a chunk
    double all = 0, most = 0;
    long long chunks = 0;
    for (size_t k = 0; k < tiles.size(); ++k) {
        all += item_cost + cost(k) * ch[k].y;
        most = std::max(most, item_cost + cost(k) * ch[k].y);
        chunks += ch[k].y;
    }
    int n = c->tc->nsm;
    if (split) {
        n = (int)std::min<long long>(n, std::max(1LL, chunks / 8));
        if (most > 0) n = std::max(1, std::min(n, (int)(all * TC_PARTS / most)));
    }
    w->n = n;
    std::vector<int> ptr(n + 1, 0);
    std::vector<int4> item;
    std::vector<int2> run;
    std::vector<unsigned char> np(std::max(c->N, 1), 0);
    double before = 0;
    int s = 0;
    auto put = [&](size_t k, int part, int a, int e) {
        item.push_back(make_int4(tiles[k].x, tiles[k].y, tiles[k].z, part));
        run.push_back(make_int2(ch[k].x + a, e - a));
        ptr[s + 1]++;
    };
    for (size_t k = 0; k < tiles.size(); ++k) {
        const double ck = cost(k);
        const int nch = ch[k].y;
        int part = 0;
        if (!split) {
            s = all > 0 ? std::max(s, std::min(n - 1, (int)((before + 0.5 * (item_cost + ck * nch)) * n / all))) : 0;
            put(k, part++, 0, nch);
        }
        for (int a = 0; split && a < nch;) {
            int e = s == n - 1 ? nch : std::min(nch, (int)std::lround((all * (s + 1) / n - before - item_cost) / ck));
            if (nch - e <= 2) e = nch;
            if (e <= a || (e < nch && e - a <= 2)) {
                ++s;
                continue;
            }
            put(k, part++, a, e);
            a = e;
            if (e < nch) ++s;
        }
        before += item_cost + ck * nch;
        w->parts = std::max(w->parts, part);
        if (split)
            for (int r = 0; r < tiles[k].z; ++r) np[c->box_ptr[tiles[k].x] + tiles[k].y + r] = (unsigned char)part;
    }
    for (int q = 0; q < n; ++q) ptr[q + 1] += ptr[q];
    CK(cudaMalloc(&w->ptr, ptr.size() * sizeof(int)));
    CK(cudaMalloc(&w->item, std::max<size_t>(item.size(), 1) * sizeof(int4)));
    CK(cudaMalloc(&w->ch, std::max<size_t>(run.size(), 1) * sizeof(int2)));
    CK(cudaMalloc(&w->np, np.size()));
    CK(cudaMemcpy(w->ptr, ptr.data(), ptr.size() * sizeof(int), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(w->item, item.data(), item.size() * sizeof(int4), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(w->ch, run.data(), run.size() * sizeof(int2), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(w->np, np.data(), np.size(), cudaMemcpyHostToDevice));
    return MLF_OK;
}

void tc_free(Ctx* c) {
    TcState* t = c->tc;
    if (!t) return;
    auto F = [](void* p) { if (p) cudaFree(p); };
    F(t->dlist); F(t->dzrow); F(t->dcbase); F(t->dchunk); F(t->derr);
    F(t->Z.hi); F(t->Z.lo); F(t->Z.rinv); F(t->M.hi); F(t->M.lo); F(t->M.rinv); F(t->xhi); F(t->xlo);
    F(t->dcmax); F(t->dcinv); F(t->drowmax); F(t->RA.rinv);
    F(t->dabase); F(t->drbase); F(t->RA.hi); F(t->RA.lo); F(t->RR.hi); F(t->RR.lo);
    F(t->dws);
    tc_slots_free(&t->near);
    tc_slots_free(&t->recv);
    tc_slots_free(&t->agg);
    delete t;
    c->tc = nullptr;
}

// FP16 operand of a matrix on the near pattern (the near field Z or the
// preconditioner M) from its box-pair blocks: per-row scales, then the rows
static void tc_operand_free(TcOperand* op) {
    if (op->hi) cudaFree(op->hi);
    if (op->lo) cudaFree(op->lo);
    if (op->rinv) cudaFree(op->rinv);
    op->hi = op->lo = nullptr;
    op->rinv = nullptr;
}

static int tc_near_operand_build(Ctx* c, const float2* blk, TcOperand* op, cudaStream_t s);

// built completely or not at all (a later call would otherwise take a half-built
// operand for a ready one)
static int tc_near_operand(Ctx* c, const float2* blk, TcOperand* op, cudaStream_t s) {
    const int st = tc_near_operand_build(c, blk, op, s);
    if (st) tc_operand_free(op);
    return st;
}

static int tc_near_operand_build(Ctx* c, const float2* blk, TcOperand* op, cudaStream_t s) {
    TcState* t = c->tc;
    const size_t bytes = (size_t)std::max<long long>(t->zrows, 1) * 128;
    CK(cudaMalloc(&op->hi, bytes));
    CK(cudaMalloc(&op->lo, bytes));
    CK(cudaMalloc(&op->rinv, (size_t)std::max(c->N, 1) * sizeof(float)));
    const int ne = (int)c->nbox_list.size();
    CK(cudaMemsetAsync(t->drowmax, 0, (size_t)c->N * sizeof(unsigned), s));
    if (ne) {
        k_blk_rowmax<<<ne, 128, 0, s>>>(c->dblk_entry, c->dnbox_list, c->dblk_off, c->dbox_ptr, blk, t->drowmax);
        k_tc_fill_zh<<<ne, 256, 0, s>>>(c->dblk_entry, c->dnbox_list, c->dblk_off, c->dbox_ptr, t->dzrow, blk,
                                        t->drowmax, static_cast<__half2*>(op->hi), static_cast<__half2*>(op->lo));
    }
    k_rinv<<<(c->N + 255) / 256, 256, 0, s>>>(c->N, t->drowmax, op->rinv);
    CK(cudaGetLastError());
    int st;
    if ((st = make_rows_map(c, &op->mhi, op->hi, t->zrows, TC_ZBOX))) return st;
    if ((st = make_rows_map(c, &op->mlo, op->lo, t->zrows, TC_ZBOX))) return st;
    return MLF_OK;
}

static int tc_setup_build(Ctx* c);

// tiles, chunk tables and the Z operand (needs the box-pair blocks); on a
// failure nothing is kept, so that the next call starts over
static int tc_setup(Ctx* c) {
    if (c->tc) return MLF_OK;
    const int st = tc_setup_build(c);
    if (st) tc_free(c);
    return st;
}

template <int MODE>
static bool tc_smem(Ctx* c) {
    return cuda_ok(c, cudaFuncSetAttribute(k_tc_gemm<MODE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)TcRing<MODE, false>::SMEM), "shared memory") &&
           cuda_ok(c, cudaFuncSetAttribute(k_tc_gemm<MODE, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)TcRing<MODE, true>::SMEM), "shared memory");
}

static int tc_setup_build(Ctx* c) {
    int st;
    if ((st = device_blocks_ready(c))) return st;
    const int nb = (int)c->box_ptr.size() - 1;
    const int ne = c->nbox_ptr[nb];
    std::vector<int4> tiles;
    for (int i = 0; i < nb; ++i) {
        const int ni = c->box_ptr[i + 1] - c->box_ptr[i];
        if (ni <= 0) continue;
        const int nt = (ni + TC_ROWS - 1) / TC_ROWS;
        const int per = ((ni + nt - 1) / nt + 15) / 16 * 16;   // rows per tile, multiple of 16
        for (int r0 = 0; r0 < ni; r0 += per) {
            const int nrow = std::min(per, ni - r0);
            if (!tc::valid_shape(128, (nrow + 15) / 16 * 16)) {
                c->err = "tensor-core near field: invalid tile shape";
                return MLF_E_STATE;
            }
            tiles.push_back(make_int4(i, r0, nrow, 0));
        }
    }
    std::vector<int> cbase(nb + 1, 0);
    std::vector<int2> chunk;
    for (int j = 0; j < nb; ++j) {
        const int j0 = c->box_ptr[j], nj = c->box_ptr[j + 1] - j0;
        cbase[j] = (int)chunk.size();
        for (int kc = 0; kc * TC_KCH_H < nj; ++kc)
            chunk.push_back(make_int2(j0 + kc * TC_KCH_H, std::min(TC_KCH_H, nj - kc * TC_KCH_H)));
    }
    cbase[nb] = (int)chunk.size();
    std::vector<int> zrow(std::max(ne, 1), 0);
    long long rows = 0;
    for (int i = 0; i < nb; ++i) {
        const int ni = c->box_ptr[i + 1] - c->box_ptr[i];
        for (int e = c->nbox_ptr[i]; e < c->nbox_ptr[i + 1]; ++e) {
            const int j = c->nbox_list[e];
            zrow[e] = (int)rows;
            rows += (long long)ni * (cbase[j + 1] - cbase[j]);
        }
    }
    if (rows >= (1LL << 31) - 256 || (long long)chunk.size() * 2 * 128 >= (1LL << 31)) {
        c->err = "tensor-core near field: operand layout exceeds 2^31 rows";
        return MLF_E_STATE;
    }
    // near chunks of each box in order
    std::vector<int2> list;
    std::vector<int> lptr(nb + 1, 0);
    for (int i = 0; i < nb; ++i) {
        const int ni = c->box_ptr[i + 1] - c->box_ptr[i];
        for (int e = c->nbox_ptr[i]; ni > 0 && e < c->nbox_ptr[i + 1]; ++e) {
            const int j = c->nbox_list[e];
            for (int k = cbase[j]; k < cbase[j + 1]; ++k) list.push_back(make_int2(k, zrow[e] + (k - cbase[j]) * ni));
        }
        lptr[i + 1] = (int)list.size();
    }
    std::vector<int2> tch;   // per tile: its first chunk in the list, chunks
    for (const int4& q : tiles) tch.push_back(make_int2(lptr[q.x], lptr[q.x + 1] - lptr[q.x]));
    int nsm = 0;
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->dev));
    TcState* t = new TcState();
    t->nsm = std::max(nsm, 1);
    c->tc = t;
    t->tiles = tiles;
    for (const int4& q : tiles) t->maxrows = std::max(t->maxrows, q.z);
    if ((st = tc_slots(c, &t->near, tiles, tch, true, 184, 2500))) return st;
    CK(cudaMalloc(&t->dlist, std::max<size_t>(list.size(), 1) * sizeof(int2)));
    CK(cudaMemcpy(t->dlist, list.data(), list.size() * sizeof(int2), cudaMemcpyHostToDevice));
    t->nchunk = (int)chunk.size();
    t->zrows = rows;
    CK(cudaMalloc(&t->dzrow, zrow.size() * sizeof(int)));
    CK(cudaMalloc(&t->dcbase, cbase.size() * sizeof(int)));
    CK(cudaMalloc(&t->dchunk, std::max<size_t>(chunk.size(), 1) * sizeof(int2)));
    CK(cudaMalloc(&t->derr, sizeof(int)));
    CK(cudaMalloc(&t->drowmax, std::max(c->N, 1) * sizeof(unsigned)));
    CK(cudaMemcpy(t->dzrow, zrow.data(), zrow.size() * sizeof(int), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(t->dcbase, cbase.data(), cbase.size() * sizeof(int), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(t->dchunk, chunk.data(), chunk.size() * sizeof(int2), cudaMemcpyHostToDevice));
    CK(cudaMemset(t->derr, 0, sizeof(int)));
    if ((st = tc_near_operand(c, c->dZblk, &t->Z, c->stream))) return st;
    if (!tc_smem<TCM_NEAR>(c) || !tc_smem<TCM_AGG>(c) || !tc_smem<TCM_RECV>(c)) return MLF_E_CUDA;
    CK(cudaStreamSynchronize(c->stream));
    return MLF_OK;
}

// X operand buffers for nrhs columns (grown on demand; maps re-encoded)
static int tc_x_buffers(Ctx* c, int nrhs) {
    TcState* t = c->tc;
    const int nct = (nrhs + TC_COLS - 1) / TC_COLS;
    const long long rows = (long long)nct * t->nchunk * 128;
    // whole column tiles, as the operand: a block that fits the one fits the other
    const size_t parts = (size_t)(t->near.parts + t->recv.parts) * c->N * nct * TC_COLS;
    if (parts > t->ws_cap) {
        if (t->dws) cudaFree(t->dws);
        t->dws = nullptr;
        t->ws_cap = 0;
        CK(cudaMalloc(&t->dws, parts * sizeof(float2)));
        t->ws_cap = parts;
    }
    if (rows <= t->xrows_cap && nct * TC_COLS <= t->cols_cap) return MLF_OK;
    auto F = [](void* p) { if (p) cudaFree(p); };
    F(t->xhi); F(t->xlo); F(t->dcmax); F(t->dcinv);
    t->xhi = t->xlo = nullptr;
    t->dcmax = nullptr;
    t->dcinv = nullptr;
    t->xrows_cap = 0;
    t->cols_cap = 0;
    CK(cudaMalloc(&t->xhi, (size_t)rows * 64));
    CK(cudaMalloc(&t->xlo, (size_t)rows * 64));
    CK(cudaMalloc(&t->dcmax, (size_t)nct * TC_COLS * sizeof(unsigned)));
    CK(cudaMalloc(&t->dcinv, (size_t)nct * TC_COLS * sizeof(float)));
    int st;
    if ((st = make_map_2d(c, &t->mxhi, t->xhi, 16, rows, 64, 16, 128, CU_TENSOR_MAP_SWIZZLE_64B))) return st;
    if ((st = make_map_2d(c, &t->mxlo, t->xlo, 16, rows, 64, 16, 128, CU_TENSOR_MAP_SWIZZLE_64B))) return st;
    t->xrows_cap = rows;
    t->cols_cap = nct * TC_COLS;
    return MLF_OK;
}

// X operand from xs (box-sorted rows, N x nrhs): per-column scales, then the packed FP16 rows
static int tc_pack_x(Ctx* c, const float2* xs, int nrhs, cudaStream_t s) {
    TcState* t = c->tc;
    const int nct = (nrhs + TC_COLS - 1) / TC_COLS;
    CK(cudaMemsetAsync(t->dcmax, 0, (size_t)nrhs * sizeof(unsigned), s));
    k_tc_colmax<<<dim3((c->N + 63) / 64, nct), 256, 0, s>>>(c->N, nrhs, xs, t->dcmax);
    k_tc_pack_xh<<<dim3(t->nchunk, nct), 256, 0, s>>>(t->nchunk, nrhs, t->dchunk, xs, t->dcmax,
                                                      static_cast<__half2*>(t->xhi), static_cast<__half2*>(t->xlo),
                                                      t->dcinv);
    return cuda_ok(c, cudaGetLastError(), "tensor-core X operand") ? MLF_OK : MLF_E_CUDA;
}

// kernel arguments common to every launch
static TcArgs tc_args(const Ctx* c, int nrhs) {
    const TcState* t = c->tc;
    TcArgs a{};
    a.nct = (nrhs + TC_COLS - 1) / TC_COLS;
    a.box_ptr = c->dbox_ptr;
    a.list = t->dlist;
    a.cbase = t->dcbase;
    a.nchunk = t->nchunk;
    a.nrhs = nrhs;
    a.cinv = t->dcinv;
    a.N = c->N;
    a.ws = t->dws;
    a.err = t->derr;
    return a;
}

// persistent grid: one CTA per SM, at most one per share and column tile
template <int MODE>
static void tc_launch(const TcState* t, const TcSlots& w, int rows, const CUtensorMap& bhi, const CUtensorMap& blo,
                      const CUtensorMap& xhi, const CUtensorMap& xlo, TcArgs a, cudaStream_t s) {
    a.nslots = w.n;
    a.slot = w.ptr;
    a.item = w.item;
    a.ch = w.ch;
    const unsigned grid = (unsigned)std::max(1, std::min(t->nsm, w.n * a.nct));
    // the pair of a tile's accumulators twice in TMEM up to 128 rows, the receive's one always
    a.nbuf = MODE == TCM_RECV || rows <= (int)TC_TMEM_COLS / 2 ? 2 : 1;
    if (rows <= TcRing<MODE, true>::ROWS)
        k_tc_gemm<MODE, true><<<grid, TC_THREADS<MODE>, TcRing<MODE, true>::SMEM, s>>>(bhi, blo, xhi, xlo, a);
    else
        k_tc_gemm<MODE, false><<<grid, TC_THREADS<MODE>, TcRing<MODE, false>::SMEM, s>>>(bhi, blo, xhi, xlo, a);
}

static dim3 tc_sum_grid(const Ctx* c, int nrhs) { return dim3((c->N + 31) / 32, (nrhs + 31) / 32); }

// the receive's parts follow the near field's
static float2* tc_recv_ws(const Ctx* c, int nrhs) { return c->tc->dws + (size_t)c->tc->near.parts * c->N * nrhs; }

// y(:, 0:nrhs) = Z_near xs + the receive of the same product on the tensor cores
// (engine 4); the X operand holds xs, packed by the product's aggregation
int device_near_tc(Ctx* c, int ld, int nrhs, double2* y, cudaStream_t s) {
    TcState* t = c->tc;
    TcArgs a = tc_args(c, nrhs);
    a.rinv = t->Z.rinv;
    tc_launch<TCM_NEAR>(t, t->near, t->maxrows, t->Z.mhi, t->Z.mlo, t->mxhi, t->mxlo, a, s);
    k_tc_sum<<<tc_sum_grid(c, nrhs), 256, 0, s>>>(c->N, nrhs, ld, c->dpos, t->near.np, t->dws, t->recv.np,
                                                  tc_recv_ws(c, nrhs), y);
    return cuda_ok(c, cudaGetLastError(), "tensor-core near field") ? MLF_OK : MLF_E_CUDA;
}

// out (FP32 columns, ld N) = M xs for the near-pattern preconditioner M, given
// as box-pair blocks (the layout of the near field's): the same kernel with M
// in place of Z, its operand layout built on first use after each rebuild of M
int device_near_pattern_tc(Ctx* c, const float2* Mblk, const float2* xs, int nrhs, float2* out, cudaStream_t s) {
    int st;
    if ((st = tc_setup(c))) return st;
    if ((st = tc_x_buffers(c, nrhs))) return st;
    TcState* t = c->tc;
    if (!t->M.hi && (st = tc_near_operand(c, Mblk, &t->M, s))) return st;
    if ((st = tc_pack_x(c, xs, nrhs, s))) return st;
    TcArgs a = tc_args(c, nrhs);
    a.rinv = t->M.rinv;
    tc_launch<TCM_NEAR>(t, t->near, t->maxrows, t->M.mhi, t->M.mlo, t->mxhi, t->mxlo, a, s);
    k_tc_sum<<<tc_sum_grid(c, nrhs), 256, 0, s>>>(c->N, nrhs, c->N, c->dpos, t->near.np, t->dws,
                                                  static_cast<const unsigned char*>(nullptr),
                                                  static_cast<const float2*>(nullptr), out);
    return cuda_ok(c, cudaGetLastError(), "tensor-core near-pattern preconditioner") ? MLF_OK : MLF_E_CUDA;
}

// Aggregation and receive operands of the leaf level from the FP32 patterns R
// (2K values per basis, box-sorted rows), built once per context:
//   RA row abase[b] + kc 2K + q = s_bq R(32 kc + u, q), u = 0..31 (bases of box
//      b), FP16 hi and lo;
//   RR row rbase[b] + kc n_b + p = conj R(p, 16 kc + u), u = 0..15 (directions),
//      TF32 hi and lo;
// zero past the box's bases / the 2K directions.
static int tc_leaf_setup(Ctx* c, const float2* R, int K2) {
    int st;
    if ((st = tc_setup(c))) return st;
    TcState* t = c->tc;
    if (t->RA.hi && t->Rsrc == R && t->K2 == K2) return MLF_OK;
    auto F = [](void* p) { if (p) cudaFree(p); };
    F(t->dabase); F(t->drbase);
    F(t->RA.hi); F(t->RA.lo); F(t->RA.rinv); F(t->RR.hi); F(t->RR.lo);
    t->dabase = t->drbase = nullptr;
    t->RA.hi = t->RA.lo = t->RR.hi = t->RR.lo = nullptr;
    t->RA.rinv = nullptr;
    t->Rsrc = nullptr;
    const int nb = (int)c->box_ptr.size() - 1;
    const int nqc = (K2 + TC_KCH - 1) / TC_KCH;
    const int nt = (K2 + TC_ROWS - 1) / TC_ROWS;
    const int per = ((K2 + nt - 1) / nt + 15) / 16 * 16;   // directions per tile, multiple of 16, <= 160
    std::vector<int4> tiles;
    std::vector<int2> tch;
    std::vector<int> abase(nb + 1, 0), rbase(nb + 1, 0);
    long long arows = 0, rrows = 0;
    for (int b = 0; b < nb; ++b) {
        const int n = c->box_ptr[b + 1] - c->box_ptr[b];
        const int nkc = (n + TC_KCH_H - 1) / TC_KCH_H;
        abase[b] = (int)arows;
        rbase[b] = (int)rrows;
        arows += (long long)nkc * K2;
        rrows += (long long)n * nqc;
        if (arows >= (1LL << 31) - 256 || rrows >= (1LL << 31) - 256) {
            c->err = "tensor-core leaf operators: operand layout exceeds 2^31 rows";
            return MLF_E_STATE;
        }
        for (int r0 = 0; r0 < K2; r0 += per) {
            const int nrow = std::min(per, K2 - r0);
            if (!tc::valid_shape(128, (nrow + 15) / 16 * 16)) {
                c->err = "tensor-core aggregation: invalid tile shape";
                return MLF_E_STATE;
            }
            tiles.push_back(make_int4(b, r0, nrow, 0));
            tch.push_back(make_int2(0, nkc));
        }
    }
    abase[nb] = (int)arows;
    rbase[nb] = (int)rrows;
    t->arows = std::min(per, K2);
    if ((st = tc_slots(c, &t->agg, tiles, tch, false, 248, 1200))) return st;
    if ((st = tc_slots(c, &t->recv, t->tiles, std::vector<int2>(t->tiles.size(), make_int2(0, nqc)), true, 279,
                       131))) return st;
    CK(cudaMalloc(&t->dabase, abase.size() * sizeof(int)));
    CK(cudaMalloc(&t->drbase, rbase.size() * sizeof(int)));
    CK(cudaMemcpy(t->dabase, abase.data(), abase.size() * sizeof(int), cudaMemcpyHostToDevice));
    CK(cudaMemcpy(t->drbase, rbase.data(), rbase.size() * sizeof(int), cudaMemcpyHostToDevice));
    const size_t ab = (size_t)std::max<long long>(arows, 1) * 128, rb = (size_t)std::max<long long>(rrows, 1) * 128;
    CK(cudaMalloc(&t->RA.hi, ab));
    CK(cudaMalloc(&t->RA.lo, ab));
    CK(cudaMalloc(&t->RA.rinv, (size_t)std::max(nb, 1) * K2 * sizeof(float)));
    CK(cudaMalloc(&t->RR.hi, rb));
    CK(cudaMalloc(&t->RR.lo, rb));
    if (nb) {
        k_tc_fill_rah<<<nb, 256, 0, c->stream>>>(K2, c->dbox_ptr, t->dabase, R, static_cast<__half2*>(t->RA.hi),
                                                 static_cast<__half2*>(t->RA.lo), t->RA.rinv);
        k_tc_fill_rr<<<nb, 256, 0, c->stream>>>(K2, c->dbox_ptr, t->drbase, R, static_cast<float*>(t->RR.hi),
                                                static_cast<float*>(t->RR.lo));
    }
    CK(cudaGetLastError());
    if ((st = make_rows_map(c, &t->RA.mhi, t->RA.hi, arows, TC_ZBOX))) return st;
    if ((st = make_rows_map(c, &t->RA.mlo, t->RA.lo, arows, TC_ZBOX))) return st;
    if ((st = make_rows_map(c, &t->RR.mhi, t->RR.hi, rrows, TC_ZBOX))) return st;
    if ((st = make_rows_map(c, &t->RR.mlo, t->RR.lo, rrows, TC_ZBOX))) return st;
    CK(cudaStreamSynchronize(c->stream));
    t->Rsrc = R;
    t->K2 = K2;
    return MLF_OK;
}

// C (leaf fields, FP32, [box][column][2K]) = R^T xs per box on the tensor
// cores.  Packs the X operand, which the near field of the same product reuses.
int device_agg_tc(Ctx* c, const float2* R, int K, const float2* xs, int nrhs, float2* C, cudaStream_t s) {
    int st;
    if ((st = tc_leaf_setup(c, R, 2 * K))) return st;
    if ((st = tc_x_buffers(c, nrhs))) return st;
    TcState* t = c->tc;
    if ((st = tc_pack_x(c, xs, nrhs, s))) return st;
    TcArgs a = tc_args(c, nrhs);
    a.zrow = t->dabase;
    a.K2 = 2 * K;
    a.C = C;
    a.rinv = t->RA.rinv;
    tc_launch<TCM_AGG>(t, t->agg, t->arows, t->RA.mhi, t->RA.mlo, t->mxhi, t->mxlo, a, s);
    return cuda_ok(c, cudaGetLastError(), "tensor-core aggregation") ? MLF_OK : MLF_E_CUDA;
}

// j facy conj(R) A per leaf box on the tensor cores, left as parts for
// device_near_tc; A the leaf fields [box][column][2K], staged raw by TMA and
// expanded in the CTA
int device_recv_tc(Ctx* c, const float2* R, int K, const float2* A, float facy, int nrhs, cudaStream_t s) {
    int st;
    const int K2 = 2 * K;
    if ((st = tc_leaf_setup(c, R, K2))) return st;
    TcState* t = c->tc;
    const int nb = (int)c->box_ptr.size() - 1;
    CUtensorMap raw;
    if ((st = make_map_2d(c, &raw, A, 2LL * K2, (long long)nb * nrhs, (long long)K2 * (long long)sizeof(float2),
                          2 * TC_KCH, TC_COLS, CU_TENSOR_MAP_SWIZZLE_128B)))
        return st;
    TcArgs a = tc_args(c, nrhs);
    a.zrow = t->drbase;
    a.K2 = K2;
    a.facy = facy;
    a.ws = tc_recv_ws(c, nrhs);
    tc_launch<TCM_RECV>(t, t->recv, t->maxrows, t->RR.mhi, t->RR.mlo, raw, raw, a, s);
    return cuda_ok(c, cudaGetLastError(), "tensor-core receive") ? MLF_OK : MLF_E_CUDA;
}

// the preconditioner's operand layout is stale once its blocks are rebuilt
void tc_drop_precond(Ctx* c) {
    TcState* t = c->tc;
    if (!t) return;
    tc_operand_free(&t->M);
}

// error flag of the tensor-core kernels since the last check (0: none)
int tc_check(Ctx* c) {
    TcState* t = c->tc;
    if (!t) return MLF_OK;
    int h = 0;
    CK(cudaMemcpy(&h, t->derr, sizeof(int), cudaMemcpyDeviceToHost));
    if (h) {
        CK(cudaMemset(t->derr, 0, sizeof(int)));
        c->err = "tensor-core near field: an mbarrier wait gave up (output skipped)";
        return MLF_E_CUDA;
    }
    return MLF_OK;
}

}  // namespace mlf
