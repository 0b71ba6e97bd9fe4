// Neighbourhood-inverse preconditioner for large neighbourhoods: a blocked,
// FP32, partially pivoted LU per leaf box.
//
// The preconditioner (mlf_precond.cu) needs, for every leaf box b, the rows of
// inv(A) that belong to b's own bases, A = Znear[S, S] over the box's near
// list S.  Its FP64 elimination works by rank-1 updates of A in global memory,
// which is fine for neighbourhoods of a few hundred unknowns but not for the
// 1500-4000 unknowns of bodies with 60-150 bases per 0.25 lambda leaf box
// (the prolate spheroid of the 722-RHS workload, the superellipsoids of the
// learned preconditioner): there the work is ~2.7 n^3 flops per box and the
// rank-1 form re-reads the whole matrix n times.
//
// This kernel solves the same system, A^T X = E_own (then M rows = X^T), with
// a right-looking blocked LU of A^T, column-major in a per-CTA slab of global
// memory (L2-resident in part):
//   for each panel of LU_P = 32 columns:
//     * panel factorisation: pivot = largest |a|^2 at or below the diagonal
//       (first row on ties), row swap, scaling, rank-1 updates, on up to eight
//       columns at a time held in shared memory (the rest of the panel is
//       updated once per eight columns); the swaps are joined to one list of
//       moved rows;
//     * moved rows, then U12 = L11^-1 A12, for the trailing columns and the
//       right-hand sides X (forward substitution on 32 x 64 tiles, four threads
//       per column with the column's rows in registers);
//     * trailing update A22 -= L21 U12 and X2 -= L21 X1 by strips of 64
//       rows: a register-blocked FP32 GEMM over 64 x 64 complex tiles (each
//       thread 2 x 8 outputs), L staged once per strip, the next U tile and
//       the current output tile loaded while the FMAs run;
//   back substitution U X = Y by blocks of 32 rows from the bottom (a small
//   triangular solve per block, then a tiled GEMM update of the rows above).
// Persistent CTAs (one or two per SM) take boxes from an atomic counter, largest
// neighbourhoods first, so large and small neighbourhoods balance over the GPU.
//
// The same kernel computes the learned preconditioner's training targets
// (mlf_learned.cu): rows of the inverse over each box's 2-ring (125-box)
// neighbourhood, the system taken from a dense Z.
//
// FP32 with partial pivoting leaves the preconditioner's rows within ~1e-5 of
// the FP64 ones (tested); a preconditioner only has to be close, and the
// solves' residual test stays FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "mlf_f32x2.cuh"
#include "mlf_internal.h"

namespace mlf {

#define CK(call)                                             \
    do {                                                     \
        if (!cuda_ok(c, (call), #call)) return MLF_E_CUDA;   \
    } while (0)

constexpr int LU_P = 32;          // panel width (= block of the back substitution)
constexpr int LU_T = 64;          // GEMM tile rows and columns
constexpr int LU_THREADS = 256;
constexpr int LU_SMEM1 = 112 * 1024, LU_SMEM2 = 64 * 1024;   // of the one-CTA-per-box kernel at one and two CTAs per SM
constexpr int LU_PANEL_SMEM = 216 * 1024, LU_PANEL_THREADS = 1024;   // of the large boxes' panels (one per SM)
constexpr int LU_BIG_GROUPS = 2;      // groups of large boxes, each in step on a stream of its own
constexpr int LU_BIG_N = 1600;        // boxes from this size on go to the many-CTA path, smaller ones ...
constexpr double LU_BIG_FACTOR = 1.0; // ... above this many CTA shares of the work that remains, or three times
                                      // as many where boxes are many (2216 of 780: 163 ms, 168 with one share)

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// d -= l u, and l = a b, in one fixed fused form: near blocks can be so badly
// conditioned that a last-place difference between two ways through the panel
// (columns at a time, CTAs of the box) would show in the inverse's third digit
__device__ __forceinline__ void sub_prod(float2& d, float2 l, float2 u) {
    d.x -= __fmaf_rn(l.x, u.x, -__fmul_rn(l.y, u.y));
    d.y -= __fmaf_rn(l.y, u.x, __fmul_rn(l.x, u.y));
}
__device__ __forceinline__ float2 prod(float2 a, float2 b) {
    return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 cinvf(float2 a) {
    const float d = a.x * a.x + a.y * a.y;
    return make_float2(a.x / d, -a.y / d);
}

__device__ __forceinline__ int bsearch_cols(const int* S, int n, int v) {
    int lo = 0, hi = n - 1;
    while (lo <= hi) {
        const int mid = (lo + hi) >> 1;
        const int s = S[mid];
        if (s == v) return mid;
        if (s < v) lo = mid + 1;
        else hi = mid - 1;
    }
    return -1;
}

// One 64-row strip of D -= Lop * Uop over K = kb, 64 columns at a time:
//   Lop(i, t) = A[(lk + t) * n + lr + r0 + i]                     (column-major panel)
//   Uop(t, j) = col(j)[uk + t],  col(q) = q < nc ? A + (ac + q) * n : X + (q - nc) * n
//   D(i, j)   = col(j)[dr + r0 + i]
// rows r0 .. r0+63 (< nrows), columns cbeg .. cend-1.  The L tile is staged
// once per strip; while a column tile is multiplied, the next tile's U values
// and the current tile's D values are already in flight (registers), so the
// loads overlap the FMAs.  Warp w owns columns 8w .. 8w+7 of a tile and each
// lane rows lane and lane + 32: the U values are warp-wide broadcasts and the
// D accesses coalesced.  The FMAs are packed over pairs of columns, in half the
// issue slots, each sum as before (inverses, scalar -> packed: 2216 boxes of 776
// unknowns 164 -> 151 ms, 504 of 790 55.8 -> 53, 824 of 2157 1155 -> 1127, 32 of
// 2014 unchanged; 128 rows a tile were slower).  The caller synchronises before;
// this ends synchronised.
// The 2-ring variant (training targets of the learned preconditioner): the
// system comes from a dense Z (complex(4), row-major N x N) over each box's
// sorted 2-ring list, and the rows go to M2 on the near pattern.  Zd null:
// the near-list variant.
struct LuRing {
    const float2* Zd = nullptr;
    int N = 0;
    const long long* off = nullptr;
    const int* len = nullptr;
    const int* bases = nullptr;
    float2* M2 = nullptr;
};

struct LuTiles {
    float2 L[LU_T][LU_P + 1];
    union {
        float2 U[2][LU_P][LU_T + 1];
        float P[2][2][LU_P][LU_T + 4];   // trailing update: real and imaginary parts apart, pairs of columns
    };
};
static_assert(sizeof(LuTiles) <= LU_SMEM2, "the one-CTA kernel's shared memory holds the tiles");

// The panel's row swaps as one move: row k0 + t gets row top[t]; row pos[t] (below
// the panel's diagonal block, -1: none) gets row from[t].
struct LuMoves {
    int top[LU_P], pos[LU_P], from[LU_P];
};

constexpr int LU_W = 8;   // columns of a panel factorised together in shared memory

struct LuShared {
    float val[32];
    int idx[32];
    int piv, sing;
    float2 u[LU_P][LU_W];
    LuMoves mv;
};

__device__ __forceinline__ float2* lu_col(float2* A, float2* X, int n, int ac, int nc, int q) {
    return q < nc ? A + (size_t)(ac + q) * n : X + (size_t)(q - nc) * n;
}

__device__ __forceinline__ void lu_strip_update(LuTiles& sm, float2* __restrict__ A, float2* __restrict__ X, int n,
                                                int kb, int lk, int lr, int uk, int dr, int ac, int nc, int r0,
                                                int nrows, int cbeg, int cend) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    constexpr int PER = LU_T * LU_P / LU_THREADS;   // U values per thread per tile (8)
#pragma unroll
    for (int e = tid; e < LU_T * LU_P; e += LU_THREADS) {
        const int t = e / LU_T, i = e - t * LU_T;          // consecutive threads: consecutive rows
        sm.L[i][t] = (t < kb && r0 + i < nrows) ? A[(size_t)(lk + t) * n + lr + r0 + i] : make_float2(0.f, 0.f);
    }
    float2 un[PER];
    auto load_u = [&](int c0) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int e = tid + k * LU_THREADS;
            const int j = e / LU_P, t = e - j * LU_P;      // consecutive threads: consecutive t of one column
            un[k] = (t < kb && c0 + j < cend) ? lu_col(A, X, n, ac, nc, c0 + j)[uk + t] : make_float2(0.f, 0.f);
        }
    };
    auto stage_u = [&](int buf) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int e = tid + k * LU_THREADS;
            const int j = e / LU_P, t = e - j * LU_P;
            sm.P[buf][0][t][j] = un[k].x;
            sm.P[buf][1][t][j] = un[k].y;
        }
    };
    load_u(cbeg);
    stage_u(0);
    __syncthreads();
    int buf = 0;
    for (int c0 = cbeg; c0 < cend; c0 += LU_T) {
        // in flight during the FMAs: the next tile's U values and this tile's D values
        if (c0 + LU_T < cend) load_u(c0 + LU_T);
        float2 d[2][8];
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const int q = c0 + 8 * w + v;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = lane + 32 * u;
                d[u][v] = (q < cend && r0 + i < nrows) ? lu_col(A, X, n, ac, nc, q)[dr + r0 + i]
                                                       : make_float2(0.f, 0.f);
            }
        }
        // the K-sum accumulates on its own and is subtracted once (the
        // in-place form rounds each product against the larger D value)
        f32x2 ax[2][4], ay[2][4];   // rows lane, lane + 32; pairs of columns
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) ax[u][v] = ay[u][v] = 0;
        for (int t = 0; t < kb; ++t) {
            const ulonglong2* px = reinterpret_cast<const ulonglong2*>(&sm.P[buf][0][t][8 * w]);
            const ulonglong2* py = reinterpret_cast<const ulonglong2*>(&sm.P[buf][1][t][8 * w]);
            const ulonglong2 x0 = px[0], x1 = px[1], y0 = py[0], y1 = py[1];
            const f32x2 bx[4] = {x0.x, x0.y, x1.x, x1.y}, by[4] = {y0.x, y0.y, y1.x, y1.y};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float2 l = sm.L[lane + 32 * u][t];
                const f32x2 lx = pk2(l.x, l.x), ly = pk2(l.y, l.y), ln = pk2(-l.y, -l.y);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    ax[u][v] = fma2(lx, bx[v], ax[u][v]);
                    ay[u][v] = fma2(lx, by[v], ay[u][v]);
                }
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    ax[u][v] = fma2(ln, by[v], ax[u][v]);
                    ay[u][v] = fma2(ly, bx[v], ay[u][v]);
                }
            }
        }
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const int q = c0 + 8 * w + v;
            if (q >= cend) continue;
            float2* col = lu_col(A, X, n, ac, nc, q);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int i = lane + 32 * u;
                const float2 x = up2(ax[u][v / 2]), y = up2(ay[u][v / 2]);
                if (r0 + i < nrows)
                    col[dr + r0 + i] = make_float2(d[u][v].x - (v & 1 ? x.y : x.x), d[u][v].y - (v & 1 ? y.y : y.x));
            }
        }
        if (c0 + LU_T < cend) stage_u(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
}

// ---- the phases of one box's solve, each executed by the CTAs part = 0 ..
// nparts-1 over disjoint pieces (one CTA: part 0 of 1, all of it)

// A^T column r = row S[r] of Z restricted to S; X = the own bases' unit columns.
// zeroed: A and X are already zero (else part 0 of 1 zeroes them first).
__device__ void lu_assemble(float2* A, float2* X, int b, int n, int nown, const int* S, const int* box_ptr,
                            const int* box_bases, const int* ia, const int* ja, const float2* Z, const LuRing& ring,
                            bool zeroed, int part, int nparts) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const size_t g0 = (size_t)part * LU_THREADS + tid, gs = (size_t)nparts * LU_THREADS;
    if (ring.Zd) {
        for (size_t e = g0; e < (size_t)n * n; e += gs) {
            const int r = (int)(e / n), pos = (int)(e - (size_t)r * n);
            A[e] = ring.Zd[(size_t)S[r] * ring.N + S[pos]];
        }
        if (!zeroed) {
            for (size_t e = g0; e < (size_t)n * nown; e += gs) X[e] = make_float2(0.f, 0.f);
            __syncthreads();
        }
    } else {
        if (!zeroed) {
            for (size_t e = g0; e < (size_t)n * n + (size_t)n * nown; e += gs) A[e] = make_float2(0.f, 0.f);
            __syncthreads();
        }
        for (int r = part * (LU_THREADS / 32) + wid; r < n; r += nparts * (LU_THREADS / 32)) {
            const int m = S[r];
            for (int q = ia[m] + lane; q < ia[m + 1]; q += 32) {
                const int pos = bsearch_cols(S, n, ja[q]);
                if (pos >= 0) A[(size_t)r * n + pos] = Z[q];
            }
        }
    }
    for (int cc = (int)g0; cc < nown; cc += (int)gs) {
        const int pos = bsearch_cols(S, n, box_bases[box_ptr[b] + cc]);
        if (pos >= 0) X[(size_t)cc * n + pos] = make_float2(1.f, 0.f);
    }
}

// Factorisation of the panel's columns js .. js+w-1 from row js down, P(i, q) =
// P[q * ld + i] with i from row js: shared memory, or the matrix itself where
// the columns do not fit.  pivot = largest |a|^2 at or below the diagonal (first
// row on ties), scaling, rank-1 updates; the row swap also on the panel's other
// columns; lanes of warp 0 keep the moves: lane t the row that has come to k0 + t
// (ct), and the t-th touched row below the diagonal block (pd) with the row that
// has come there (cd).  Returns false when singular.
template <int NT>
__device__ bool lu_columns(LuShared& sh, float2* P, size_t ld, float2* A, int n, int k0, int kb, int js, int w, int& ct,
                           int& pd, int& cd, int& nd) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, m = n - js;
    for (int j = 0; j < w; ++j) {
        float best = -1.f;
        int bi = m;
        const float2* colj = P + j * ld;
        for (int i = j + tid; i < m; i += NT) {
            const float2 a = colj[i];
            const float v = __fmaf_rn(a.x, a.x, __fmul_rn(a.y, a.y));
            if (v > best) { best = v; bi = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { sh.val[wid] = best; sh.idx[wid] = bi; }
        __syncthreads();
        if (wid == 0) {
            best = lane < NT / 32 ? sh.val[lane] : -1.f;
            bi = lane < NT / 32 ? sh.idx[lane] : m;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (lane == 0) {
                sh.piv = bi;
                sh.sing = !(best > 0.f) || bi >= m;
            }
            const int row = js + j, pv = js + bi;   // rows of the matrix that change places
            if (bi < m && pv != row) {
                const int tr = row - k0;
                const int mine = __shfl_sync(0xffffffffu, ct, tr);
                if (pv < k0 + LU_P) {
                    const int other = __shfl_sync(0xffffffffu, ct, pv - k0);
                    if (lane == tr) ct = other;
                    if (lane == pv - k0) ct = mine;
                } else {
                    unsigned at = __ballot_sync(0xffffffffu, lane < nd && pd == pv);
                    if (!at) {
                        if (lane == nd) { pd = pv; cd = pv; }
                        at = 1u << nd;
                        ++nd;
                    }
                    const int q = __ffs(at) - 1, other = __shfl_sync(0xffffffffu, cd, q);
                    if (lane == q) cd = mine;
                    if (lane == tr) ct = other;
                }
            }
        }
        __syncthreads();
        if (sh.sing) return false;
        const int pv = sh.piv;
        if (pv != j) {
            // threads: the w columns at hand, then the panel's others in place
            if (tid < w) {
                float2* col = P + tid * ld;
                const float2 t = col[j];
                col[j] = col[pv];
                col[pv] = t;
            } else if (tid >= 32 && tid < 32 + kb) {
                const int c = k0 + tid - 32;
                if (c < js || c >= js + w) {
                    float2* col = A + (size_t)c * n + js;
                    const float2 t = col[j];
                    col[j] = col[pv];
                    col[pv] = t;
                }
            }
            __syncthreads();
        }
        const float2 dinv = cinvf(P[j * ld + j]);
        float2 u[LU_W];
#pragma unroll
        for (int q = 1; q < LU_W; ++q)
            if (j + q < w) u[q] = P[(j + q) * ld + j];
        for (int i = j + 1 + tid; i < m; i += NT) {
            const float2 l = prod(P[j * ld + i], dinv);
            P[j * ld + i] = l;
#pragma unroll
            for (int q = 1; q < LU_W; ++q)
                if (j + q < w) {
                    float2 d = P[(j + q) * ld + i];
                    sub_prod(d, l, u[q]);
                    P[(j + q) * ld + i] = d;
                }
        }
        __syncthreads();
    }
    return true;
}

// Panel factorisation of columns k0 .. k0+kb-1 (one CTA of NT threads): up to
// LU_W columns at a time in `buf` (cap values), then the panel's later columns
// updated by all of them at once.  The moves of the rows go to mv; the trailing
// columns and X are moved by lu_u12.  Returns false when singular.
template <int NT>
__device__ bool lu_panel(LuShared& sh, float2* buf, int cap, float2* A, int n, int k0, int kb, LuMoves* mv) {
    const int tid = threadIdx.x, lane = tid & 31;
    int ct = k0 + lane, pd = -1, cd = -1, nd = 0;
    for (int js = k0; js < k0 + kb;) {
        const int m = n - js, fit = cap / m;
        const bool in = fit > 0;
        const int w = min(k0 + kb - js, in ? min(LU_W, fit) : LU_W);
        float2* P = in ? buf : A + (size_t)js * n + js;
        const size_t ld = in ? m : n;
        if (in) {
            for (int q = 0; q < w; ++q)
                for (int i = tid; i < m; i += NT) buf[(size_t)q * m + i] = A[(size_t)(js + q) * n + js + i];
            __syncthreads();
        }
        const bool ok = in ? lu_columns<NT>(sh, buf, m, A, n, k0, kb, js, w, ct, pd, cd, nd)
                           : lu_columns<NT>(sh, P, ld, A, n, k0, kb, js, w, ct, pd, cd, nd);
        if (!ok) return false;
        const int c0 = js + w, nr = k0 + kb - c0;   // the panel's later columns
        if (nr > 0) {
            // their rows js .. js+w-1: forward substitution, a thread per column
            if (tid < nr) {
                float2* col = A + (size_t)(c0 + tid) * n + js;
                for (int r = 0; r < w; ++r) {
                    float2 v = col[r];
                    for (int t = 0; t < r; ++t) sub_prod(v, P[t * ld + r], sh.u[tid][t]);
                    sh.u[tid][r] = v;
                    col[r] = v;
                }
            }
            __syncthreads();
            for (int i = w + tid; i < m; i += NT) {
                float2 l[LU_W];
#pragma unroll
                for (int t = 0; t < LU_W; ++t) l[t] = t < w ? P[t * ld + i] : make_float2(0.f, 0.f);
                for (int q0 = 0; q0 < nr; q0 += 8) {
                    float2 d[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q0 + q < nr) d[q] = A[(size_t)(c0 + q0 + q) * n + js + i];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q0 + q < nr) {
#pragma unroll
                            for (int t = 0; t < LU_W; ++t)
                                if (t < w) sub_prod(d[q], l[t], sh.u[q0 + q][t]);
                            A[(size_t)(c0 + q0 + q) * n + js + i] = d[q];
                        }
                }
            }
        }
        if (in)
            for (int q = 0; q < w; ++q)
                for (int i = tid; i < m; i += NT) A[(size_t)(js + q) * n + js + i] = buf[(size_t)q * m + i];
        __syncthreads();   // the columns are read again, buf is filled again
        js += w;
    }
    if (tid < 32) {
        mv->top[lane] = ct;
        mv->pos[lane] = lane < nd ? pd : -1;
        mv->from[lane] = cd;
    }
    return true;
}

// The panel's moves of rows, then U12 = L11^-1 A12 (and X), over the column tiles
// part, part + nparts, ... of the trailing columns and X.  Unit lower L11 in
// shared memory; a warp takes eight columns, four threads each, thread g of a
// column holding the rows g, g + 4, ... in registers: row r is passed on by a
// shuffle, and every row below subtracts its product at once.
__device__ void lu_u12(LuTiles& sm, float2* A, float2* X, int n, int nown, int k0, int kb, const LuMoves* mv, int part,
                       int nparts) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int nc = n - k0 - kb, ncols = nc + nown;
    for (int e = tid; e < LU_P * LU_P; e += LU_THREADS) {
        const int t = e / LU_P, r = e - t * LU_P;
        sm.L[r][t] = (r < kb && t < kb) ? A[(size_t)(k0 + t) * n + k0 + r] : make_float2(0.f, 0.f);
    }
    const int top = mv->top[lane], pos = mv->pos[lane], from = mv->from[lane];   // every warp: lane t the t-th move
    __syncthreads();
    for (int c0 = part * LU_T; c0 < ncols; c0 += nparts * LU_T) {
        // rows to come to the top, and to below, of 64 columns; a warp takes a column
#pragma unroll
        for (int u = 0; u < LU_T / (LU_THREADS / 32); ++u) {
            const int j = w + u * (LU_THREADS / 32);
            float2 a = make_float2(0.f, 0.f), d = a;
            if (c0 + j < ncols) {
                const float2* col = lu_col(A, X, n, k0 + kb, nc, c0 + j);
                if (lane < kb) a = col[top];
                if (pos >= 0) d = col[from];
            }
            sm.U[0][lane][j] = a;
            sm.U[1][lane][j] = d;
        }
        __syncthreads();
        {
            const int g = lane >> 3, j = 8 * w + (lane & 7);
            float2 v[LU_P / 4];
#pragma unroll
            for (int q = 0; q < LU_P / 4; ++q) v[q] = sm.U[0][4 * q + g][j];
#pragma unroll
            for (int r = 0; r < LU_P - 1; ++r) {
                const float2 own = v[r / 4];
                const float2 x = make_float2(__shfl_sync(0xffffffffu, own.x, (lane & 7) + 8 * (r & 3)),
                                             __shfl_sync(0xffffffffu, own.y, (lane & 7) + 8 * (r & 3)));
#pragma unroll
                for (int q = r / 4; q < LU_P / 4; ++q)
                    if (4 * q + g > r) sub_prod(v[q], sm.L[4 * q + g][r], x);
            }
#pragma unroll
            for (int q = 0; q < LU_P / 4; ++q) sm.U[0][4 * q + g][j] = v[q];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < LU_T / (LU_THREADS / 32); ++u) {
            const int j = w + u * (LU_THREADS / 32);
            if (c0 + j < ncols) {
                float2* col = lu_col(A, X, n, k0 + kb, nc, c0 + j);
                if (lane < kb) col[k0 + lane] = sm.U[0][lane][j];
                if (pos >= 0) col[pos] = sm.U[1][lane][j];
            }
        }
        __syncthreads();
    }
}

// back substitution of block k0 (rows k0 .. k0+kb-1 of X, U11 from A) over the
// X column tiles part, part + nparts, ...
__device__ void lu_back_block(LuTiles& sm, const float2* A, float2* X, int n, int nown, int k0, int kb, int part,
                              int nparts) {
    const int tid = threadIdx.x;
    for (int e = tid; e < LU_P * LU_P; e += LU_THREADS) {
        const int t = e / LU_P, r = e - t * LU_P;
        sm.L[r][t] = (r < kb && t < kb) ? A[(size_t)(k0 + t) * n + k0 + r] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    for (int c0 = part * LU_T; c0 < nown; c0 += nparts * LU_T) {
        // a 32 x 64 tile of X in shared memory, backward substitution per column
        for (int e = tid; e < LU_T * LU_P; e += LU_THREADS) {
            const int j = e / LU_P, t = e - j * LU_P;
            sm.U[0][t][j] = (t < kb && c0 + j < nown) ? X[(size_t)(c0 + j) * n + k0 + t] : make_float2(0.f, 0.f);
        }
        __syncthreads();
        if (tid < LU_T) {
            for (int r = kb - 1; r >= 0; --r) {
                float2 acc = sm.U[0][r][tid];
                for (int t = r + 1; t < kb; ++t) {
                    const float2 u = sm.L[r][t], x = sm.U[0][t][tid];
                    acc.x -= u.x * x.x - u.y * x.y;
                    acc.y -= u.x * x.y + u.y * x.x;
                }
                sm.U[0][r][tid] = cmulf(acc, cinvf(sm.L[r][r]));
            }
        }
        __syncthreads();
        for (int e = tid; e < LU_T * LU_P; e += LU_THREADS) {
            const int j = e / LU_P, t = e - j * LU_P;
            if (t < kb && c0 + j < nown) X[(size_t)(c0 + j) * n + k0 + t] = sm.U[0][t][j];
        }
        __syncthreads();
    }
}

// rows of the own bases: M[ia[g] + j] = X(j, own index) over the near list,
// or (2-ring) the entries of the near pattern inside the ring list
__device__ void lu_extract(const float2* X, int b, int n, int nown, const int* S, const int* box_ptr,
                           const int* box_bases, const int* ia, const int* ja, double2* M, const LuRing& ring,
                           int part, int nparts) {
    for (int cc = part; cc < nown; cc += nparts) {
        const int g = box_bases[box_ptr[b] + cc];
        const float2* col = X + (size_t)cc * n;
        if (ring.Zd) {
            for (int q = ia[g] + threadIdx.x; q < ia[g + 1]; q += LU_THREADS) {
                const int pos = bsearch_cols(S, n, ja[q]);
                ring.M2[q] = pos >= 0 ? col[pos] : make_float2(0.f, 0.f);
            }
        } else {
            double2* row = M + ia[g];
            for (int j = threadIdx.x; j < n; j += LU_THREADS) row[j] = make_double2((double)col[j].x, (double)col[j].y);
        }
    }
}

__device__ __forceinline__ void lu_box(int b, const int* box_ptr, const int* ia, const LuRing& ring, int box0,
                                       int& n, int& nown, const int*& S, const int* ja) {
    const int m0 = box0;
    nown = box_ptr[b + 1] - box_ptr[b];
    // the neighbourhood: the near list (the CSR row of the box's bases) or the 2-ring list
    n = ring.Zd ? ring.len[b] : ia[m0 + 1] - ia[m0];
    S = ring.Zd ? ring.bases + ring.off[b] : ja + ia[m0];
}

// One CTA per box, persistent: CTAs take boxes from an atomic counter in the
// given order (largest neighbourhoods first).
__global__ void __launch_bounds__(LU_THREADS, 2)
    k_nbhd_lu32(int nb, const int* __restrict__ box_ptr, const int* __restrict__ box_bases,
                const int* __restrict__ ia, const int* __restrict__ ja, const float2* __restrict__ Z, size_t slab,
                float2* __restrict__ work, double2* __restrict__ M, const int* __restrict__ order,
                int* __restrict__ next_box, int* __restrict__ bad, const LuRing ring, int smem) {
    extern __shared__ __align__(16) unsigned char lu_smem[];   // a panel's columns, or the tiles
    __shared__ LuShared sh;
    __shared__ int s_b;
    LuTiles& tiles = *reinterpret_cast<LuTiles*>(lu_smem);
    const int tid = threadIdx.x;
    float2* A = work + (size_t)blockIdx.x * slab;
    for (;;) {
        if (tid == 0) {
            const int k = atomicAdd(next_box, 1);
            s_b = k < nb ? order[k] : -1;      // largest neighbourhoods first
        }
        __syncthreads();
        const int b = s_b;
        if (b < 0) break;
        int n, nown;
        const int* S;
        lu_box(b, box_ptr, ia, ring, box_bases[box_ptr[b]], n, nown, S, ja);
        float2* X = A + (size_t)n * n;
        lu_assemble(A, X, b, n, nown, S, box_ptr, box_bases, ia, ja, Z, ring, false, 0, 1);
        __syncthreads();
        bool ok = true;
        for (int k0 = 0; k0 < n && ok; k0 += LU_P) {
            const int kb = min(LU_P, n - k0);
            ok = lu_panel<LU_THREADS>(sh, reinterpret_cast<float2*>(lu_smem), smem / (int)sizeof(float2), A, n, k0, kb,
                                      &sh.mv);
            if (!ok) break;
            __syncthreads();   // the moves
            lu_u12(tiles, A, X, n, nown, k0, kb, &sh.mv, 0, 1);
            // trailing update: rows k0+kb.. of the trailing columns and of X
            const int nrows = n - k0 - kb, nc = nrows;
            for (int r0 = 0; r0 < nrows; r0 += LU_T)
                lu_strip_update(tiles, A, X, n, kb, k0, k0 + kb, k0, k0 + kb, k0 + kb, nc, r0, nrows, 0, nc + nown);
        }
        if (!ok) {
            if (tid == 0) atomicMin(bad, b + 1);
            __syncthreads();
            continue;
        }
        // back substitution U X = Y, blocks of LU_P rows from the bottom
        for (int k0 = ((n - 1) / LU_P) * LU_P; k0 >= 0; k0 -= LU_P) {
            const int kb = min(LU_P, n - k0);
            lu_back_block(tiles, A, X, n, nown, k0, kb, 0, 1);
            // rows 0..k0-1 of X -= U(0..k0-1, k0..k0+kb-1) X(k0..k0+kb-1)
            for (int r0 = 0; r0 < k0; r0 += LU_T) lu_strip_update(tiles, A, X, n, kb, k0, 0, k0, 0, 0, 0, r0, k0, 0, nown);
        }
        lu_extract(X, b, n, nown, S, box_ptr, box_bases, ia, ja, M, ring, 0, 1);
        __syncthreads();
    }
}

// ---- large boxes on many CTAs: the same phases as kernels over a group of boxes
// in step, a launch per phase and panel for all of them (blockIdx.y = box; a box
// that is smaller, or singular, *sing set by its panel, has nothing to do)

struct LuBig {
    int b, n, nown;
    const int* S;      // device pointer into ja or the 2-ring lists
    float2* A;
    float2* X;
    LuMoves* mv;       // of the current panel
    int* sing;
};

__device__ __forceinline__ bool lu_idle(const LuBig& g, int k0) {
    return k0 >= g.n || *reinterpret_cast<volatile int*>(g.sing);
}

__global__ void __launch_bounds__(LU_THREADS) k_lub_assemble(const LuBig* __restrict__ gs,
                                                             const int* __restrict__ box_ptr,
                                                             const int* __restrict__ box_bases,
                                                             const int* __restrict__ ia, const int* __restrict__ ja,
                                                             const float2* __restrict__ Z, const LuRing ring) {
    const LuBig g = gs[blockIdx.y];
    lu_assemble(g.A, g.X, g.b, g.n, g.nown, g.S, box_ptr, box_bases, ia, ja, Z, ring, true, blockIdx.x, gridDim.x);
}

__global__ void __launch_bounds__(LU_PANEL_THREADS) k_lub_panel(const LuBig* __restrict__ gs, int k0,
                                                                int* __restrict__ bad) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    __shared__ LuShared sh;
    const LuBig g = gs[blockIdx.y];
    if (lu_idle(g, k0)) return;
    if (!lu_panel<LU_PANEL_THREADS>(sh, reinterpret_cast<float2*>(lu_smem), LU_PANEL_SMEM / (int)sizeof(float2), g.A, g.n,
                                    k0, min(LU_P, g.n - k0), g.mv) &&
        threadIdx.x == 0) {
        *g.sing = 1;
        atomicMin(bad, g.b + 1);
    }
}

__global__ void __launch_bounds__(LU_THREADS) k_lub_u12(const LuBig* __restrict__ gs, int k0) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const LuBig g = gs[blockIdx.y];
    if (lu_idle(g, k0)) return;
    lu_u12(*reinterpret_cast<LuTiles*>(lu_smem), g.A, g.X, g.n, g.nown, k0, min(LU_P, g.n - k0), g.mv, blockIdx.x,
           gridDim.x);
}

// trailing update: CTA (strip blockIdx.x % nstrip, column chunk blockIdx.x / nstrip of cw columns)
__global__ void __launch_bounds__(LU_THREADS, 2) k_lub_trail(const LuBig* __restrict__ gs, int k0, int nstrip, int cw) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const LuBig g = gs[blockIdx.y];
    if (lu_idle(g, k0)) return;
    const int n = g.n, kb = min(LU_P, n - k0);
    const int nrows = n - k0 - kb, nc = nrows, ncols = nc + g.nown;
    const int r0 = blockIdx.x % nstrip * LU_T, cb = blockIdx.x / nstrip * cw;
    if (r0 >= nrows || cb >= ncols) return;
    lu_strip_update(*reinterpret_cast<LuTiles*>(lu_smem), g.A, g.X, n, kb, k0, k0 + kb, k0, k0 + kb, k0 + kb, nc, r0,
                    nrows, cb, min(ncols, cb + cw));
}

__global__ void __launch_bounds__(LU_THREADS) k_lub_back(const LuBig* __restrict__ gs, int k0) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const LuBig g = gs[blockIdx.y];
    if (lu_idle(g, k0)) return;
    lu_back_block(*reinterpret_cast<LuTiles*>(lu_smem), g.A, g.X, g.n, g.nown, k0, min(LU_P, g.n - k0), blockIdx.x,
                  gridDim.x);
}

// rows 0..k0-1 of X -= U(0..k0-1, block k0) X(block k0): CTA per (strip, 64 X columns)
__global__ void __launch_bounds__(LU_THREADS, 2) k_lub_back_upd(const LuBig* __restrict__ gs, int k0, int nstrip) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const LuBig g = gs[blockIdx.y];
    if (lu_idle(g, k0)) return;
    const int kb = min(LU_P, g.n - k0);
    const int r0 = blockIdx.x % nstrip * LU_T, cb = blockIdx.x / nstrip * LU_T;
    if (r0 >= k0 || cb >= g.nown) return;
    lu_strip_update(*reinterpret_cast<LuTiles*>(lu_smem), g.A, g.X, g.n, kb, k0, 0, k0, 0, 0, 0, r0, k0, cb,
                    min(g.nown, cb + LU_T));
}

__global__ void __launch_bounds__(LU_THREADS) k_lub_extract(const LuBig* __restrict__ gs,
                                                            const int* __restrict__ box_ptr,
                                                            const int* __restrict__ box_bases,
                                                            const int* __restrict__ ia, const int* __restrict__ ja,
                                                            double2* __restrict__ M, const LuRing ring) {
    const LuBig g = gs[blockIdx.y];
    if (lu_idle(g, 0)) return;
    lu_extract(g.X, g.b, g.n, g.nown, g.S, box_ptr, box_bases, ia, ja, M, ring, blockIdx.x, gridDim.x);
}

// A group of large boxes, in step, on stream s: ng boxes of at most n unknowns and
// nown own ones, their slabs and `sing` flags zero.
static int big_boxes_launch(Ctx* c, const LuRing& ring, const LuBig* gs, int ng, int n, int nown, int* bad,
                            cudaStream_t s) {
    const size_t tiles = sizeof(LuTiles);
    const unsigned ga = (unsigned)std::min<long long>(std::max(1, 8192 / ng),
                                                      ((long long)n * n + LU_THREADS - 1) / LU_THREADS);
    k_lub_assemble<<<dim3(ga, ng), LU_THREADS, 0, s>>>(gs, c->dbox_ptr, c->dperm, c->dia, c->dja, c->dZ, ring);
    for (int k0 = 0; k0 < n; k0 += LU_P) {
        const int kb = std::min(LU_P, n - k0);
        const int nrows = n - k0 - kb, ncols = nrows + nown + LU_P;   // a smaller box's panel may be its last, narrower
        k_lub_panel<<<dim3(1, ng), LU_PANEL_THREADS, LU_PANEL_SMEM, s>>>(gs, k0, bad);
        k_lub_u12<<<dim3((ncols + LU_T - 1) / LU_T, ng), LU_THREADS, tiles, s>>>(gs, k0);
        if (nrows <= 0) continue;
        const int nstrip = (nrows + LU_T - 1) / LU_T;
        const int cw = std::max(LU_T, (ncols + 15) / 16 / LU_T * LU_T + LU_T);   // up to 16 chunks
        const int nchunk = (ncols + cw - 1) / cw;
        k_lub_trail<<<dim3(nstrip * nchunk, ng), LU_THREADS, tiles, s>>>(gs, k0, nstrip, cw);
    }
    const int xt = (nown + LU_T - 1) / LU_T;
    for (int k0 = ((n - 1) / LU_P) * LU_P; k0 >= 0; k0 -= LU_P) {
        k_lub_back<<<dim3(xt, ng), LU_THREADS, tiles, s>>>(gs, k0);
        if (k0 > 0) k_lub_back_upd<<<dim3(k0 / LU_T * xt + xt, ng), LU_THREADS, tiles, s>>>(gs, k0, k0 / LU_T + 1);
    }
    k_lub_extract<<<dim3(std::max(nown, 1), ng), LU_THREADS, 0, s>>>(gs, c->dbox_ptr, c->dperm, c->dia, c->dja, c->dMinv,
                                                                    ring);
    return cuda_ok(c, cudaGetLastError(), "large-box LU") ? MLF_OK : MLF_E_CUDA;
}

// Every box's rows of the inverse over its neighbourhood: ring null: the near
// list, into c->dMinv (near CSR pattern, allocated by the caller); ring given:
// the 2-ring lists (len[b] unknowns and offset off[b] each, host copies), into
// ring->M2.  *bad_box as mlf_nearinv.
//
// A box's elimination costs ~n^3.  The persistent kernel gives each box one
// CTA, so a box whose work exceeds a few average CTA shares of the rest would
// set the finishing time alone (on the 722-RHS workload's spheroid the
// largest neighbourhoods, 5648 unknowns, took most of the set-up).  Those
// boxes, largest first, run instead on many CTAs each (k_lub_*), in groups on
// side streams concurrently with the persistent kernel over the others: two
// groups, so that one's panels (a CTA per box) run beside the other's updates.
static int blocked_inverse_rows(Ctx* c, int nownmax, const LuRing* ring, const int* ring_len,
                                const long long* ring_off, int* bad_box) {
    DevScope ds;
    const int nb = (int)c->box_ptr.size() - 1;
    int nsm = 0;
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->dev));
    // boxes by decreasing neighbourhood size, so that the largest do not finish last
    auto nsize = [&](int b) { return ring ? ring_len[b] : c->near_ptr[b + 1] - c->near_ptr[b]; };
    std::vector<int> order(nb);
    for (int b = 0; b < nb; ++b) order[b] = b;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b2) { return nsize(a) > nsize(b2); });
    // the large boxes: a prefix of the order.  On many CTAs a box takes 1.3 ms at
    // 2200 unknowns, 2.2 ms a box with one CTA on each SM, so boxes from LU_BIG_N
    // on go there (122 880-RWG spheroid, 824 boxes of 2160 on average: its 16
    // largest there 1.85 s, 120 1.35 s, all 1.08 s), and smaller ones above one
    // CTA share of the remaining work (504 boxes of 790: three shares, 16 boxes,
    // 67 ms; one share, 72 boxes, 57 ms)
    std::vector<double> tail(nb + 1, 0.0);
    for (int k = nb - 1; k >= 0; --k) tail[k] = tail[k + 1] + std::pow((double)nsize(order[k]), 3.0);
    const double factor = nb >= 4 * nsm ? 3 * LU_BIG_FACTOR : LU_BIG_FACTOR;
    int nbig = 0;
    while (c->lu_big_min > 0 && nbig < nb && nsize(order[nbig]) >= c->lu_big_min &&
           (nsize(order[nbig]) >= LU_BIG_N ||
            std::pow((double)nsize(order[nbig]), 3.0) > factor * tail[nbig] / (2.0 * nsm)))
        ++nbig;
    const int nsmall = nb - nbig;
    int *dctr = nullptr, *dbad = nullptr, *dorder = nullptr;
    CK(ds.alloc(&dorder, std::max(nsmall, 1) * sizeof(int)));
    if (nsmall) CK(cudaMemcpyAsync(dorder, order.data() + nbig, nsmall * sizeof(int), cudaMemcpyHostToDevice, c->stream));
    CK(ds.alloc(&dctr, 2 * sizeof(int)));
    dbad = dctr + 1;
    const int init[2] = {0, 0x7fffffff};
    CK(cudaMemcpyAsync(dctr, init, sizeof(init), cudaMemcpyHostToDevice, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    const LuRing none{};
    const LuRing& rg = ring ? *ring : none;
    // limits of the kernels, the same for every context
    CK(cudaFuncSetAttribute(k_nbhd_lu32, cudaFuncAttributeMaxDynamicSharedMemorySize, LU_SMEM1));
    CK(cudaFuncSetAttribute(k_lub_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, LU_PANEL_SMEM));
    for (const void* k : {(const void*)k_lub_u12, (const void*)k_lub_trail, (const void*)k_lub_back,
                          (const void*)k_lub_back_upd})
        CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LuTiles)));
    // large boxes: their streams, and slabs for as many at a time as a quarter of
    // the free memory holds (all, but for the largest bodies)
    const int ngroup = std::min(nbig, LU_BIG_GROUPS);
    std::vector<cudaStream_t> bs(ngroup, nullptr);
    std::vector<float2*> bslab(ngroup, nullptr);
    std::vector<LuBig*> bdesc(ngroup, nullptr);
    std::vector<LuMoves*> bmv(ngroup, nullptr);
    int* bsing = nullptr;
    int per = 0;              // boxes of a group in step at a time
    size_t bslab_el = 0;
    int st = MLF_OK;
    if (nbig) {
        const int n0 = nsize(order[0]);
        bslab_el = (size_t)n0 * n0 + (size_t)n0 * nownmax;
        size_t fr = 0, tot = 0;
        CK(cudaMemGetInfo(&fr, &tot));
        per = (int)std::max<size_t>(1, std::min<size_t>((nbig + ngroup - 1) / ngroup,
                                                        fr / 4 / ngroup / (bslab_el * sizeof(float2))));
        if (!cuda_ok(c, ds.alloc(&bsing, (size_t)ngroup * per * sizeof(int)), "large-box scratch")) st = MLF_E_CUDA;
        for (int q = 0; q < ngroup && !st; ++q)
            if (!cuda_ok(c, ds.alloc(&bslab[q], per * bslab_el * sizeof(float2)), "large-box slabs") ||
                !cuda_ok(c, ds.alloc(&bdesc[q], per * sizeof(LuBig)), "large-box scratch") ||
                !cuda_ok(c, ds.alloc(&bmv[q], per * sizeof(LuMoves)), "large-box scratch") ||
                !cuda_ok(c, cudaStreamCreateWithFlags(&bs[q], cudaStreamNonBlocking), "large-box stream"))
                st = MLF_E_CUDA;
    }
    // the persistent kernel over the other boxes, the slabs within half of the free
    // device memory: two CTAs per SM, but one with more of its panel in shared
    // memory where boxes are few (504 boxes of 790 unknowns: 82 ms with two, 67 with
    // one; 2216 boxes: 163 and 263)
    if (nsmall && !st) {
        const int ns0 = nsize(order[nbig]);
        const size_t slab = (size_t)ns0 * ns0 + (size_t)ns0 * nownmax;
        size_t fr = 0, tot = 0;
        float2* work = nullptr;
        if (!cuda_ok(c, cudaMemGetInfo(&fr, &tot), "cudaMemGetInfo")) {
            st = MLF_E_CUDA;
        } else {
            const size_t cap = (fr / 2) / (slab * sizeof(float2));
            const int per_sm = nsmall >= 4 * nsm ? 2 : 1, smem = per_sm == 2 ? LU_SMEM2 : LU_SMEM1;
            const int grid = (int)std::max<size_t>(1, std::min<size_t>({(size_t)per_sm * nsm, (size_t)nsmall, cap}));
            if (!cuda_ok(c, ds.alloc(&work, slab * grid * sizeof(float2)), "neighbourhood LU slabs")) {
                st = MLF_E_CUDA;
            } else {
                k_nbhd_lu32<<<grid, LU_THREADS, smem, c->stream>>>(nsmall, c->dbox_ptr, c->dperm, c->dia, c->dja, c->dZ,
                                                                slab, work, c->dMinv, dorder, dctr, dbad, rg, smem);
                if (!cuda_ok(c, cudaGetLastError(), "neighbourhood LU")) st = MLF_E_CUDA;
            }
        }
    }
    // boxes dealt to the groups in turn, largest first; a group's next lot follows on its stream
    for (int k0 = 0; k0 < nbig && !st; k0 += ngroup * per) {
        for (int q = 0; q < ngroup && !st; ++q) {
            std::vector<LuBig> g;
            int ng_own = 0;
            for (int k = k0 + q; k < nbig && (int)g.size() < per; k += ngroup) {
                const int b = order[k], i = (int)g.size(), n = nsize(b), nown = c->box_ptr[b + 1] - c->box_ptr[b];
                const int* S = ring ? ring->bases + ring_off[b] : c->dja + c->ia[c->box_bases[c->box_ptr[b]]];
                float2* A = bslab[q] + i * bslab_el;
                g.push_back(LuBig{b, n, nown, S, A, A + (size_t)n * n, bmv[q] + i, bsing + (size_t)q * per + i});
                ng_own = std::max(ng_own, nown);
            }
            if (g.empty()) continue;
            if (!cuda_ok(c, cudaStreamSynchronize(bs[q]), "large-box LU") ||   // the lot before has read its descriptors
                !cuda_ok(c, cudaMemcpyAsync(bdesc[q], g.data(), g.size() * sizeof(LuBig), cudaMemcpyHostToDevice, bs[q]),
                         "large-box descriptors") ||
                !cuda_ok(c, cudaMemsetAsync(bsing + (size_t)q * per, 0, g.size() * sizeof(int), bs[q]), "memset") ||
                !cuda_ok(c, cudaMemsetAsync(bslab[q], 0, g.size() * bslab_el * sizeof(float2), bs[q]), "memset"))
                st = MLF_E_CUDA;
            else
                st = big_boxes_launch(c, rg, bdesc[q], (int)g.size(), g[0].n, ng_own, dbad, bs[q]);
        }
    }
    for (int q = 0; q < ngroup; ++q) {
        if (!bs[q]) continue;
        if (!cuda_ok(c, cudaStreamSynchronize(bs[q]), "large-box LU") && !st) st = MLF_E_CUDA;
        cudaStreamDestroy(bs[q]);
    }
    if (st) {
        cudaStreamSynchronize(c->stream);   // the persistent kernel, if launched, ends before its slabs go
        return st;
    }
    int hbad = 0;
    CK(cudaMemcpyAsync(&hbad, dbad, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    *bad_box = hbad == 0x7fffffff ? 0 : hbad;
    c->lu_big_last = nbig;
    return MLF_OK;
}

int nbhd_inverse_lu32(Ctx* c, int nownmax, int* bad_box) {
    return blocked_inverse_rows(c, nownmax, nullptr, nullptr, nullptr, bad_box);
}

int ring_inverse_lu32(Ctx* c, const float2* Zd, const long long* off, const int* len, const int* bases,
                      const std::vector<int>& len_host, const std::vector<long long>& off_host, int nownmax,
                      float2* M2, int* bad_box) {
    LuRing r;
    r.Zd = Zd;
    r.N = c->N;
    r.off = off;
    r.len = len;
    r.bases = bases;
    r.M2 = M2;
    return blocked_inverse_rows(c, nownmax, &r, len_host.data(), off_host.data(), bad_box);
}

}  // namespace mlf

using namespace mlf;

extern "C" int mlf_set_lu_split(mlf_ctx* h, int min_unknowns) {
    if (!h || min_unknowns < 0) return MLF_E_ARG;
    h->c.lu_big_min = min_unknowns;
    return MLF_OK;
}

extern "C" int mlf_get_lu_split(mlf_ctx* h, int* min_unknowns, int* last_big_boxes) {
    if (!h) return MLF_E_ARG;
    if (min_unknowns) *min_unknowns = h->c.lu_big_min;
    if (last_big_boxes) *last_big_boxes = h->c.lu_big_last;
    return MLF_OK;
}
