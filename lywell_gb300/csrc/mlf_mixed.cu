// Mixed-precision solve: FP32 MLFMA matvec inside an FP64 iterative-refinement
// loop.  (An addition of this library: the reference runs its whole matvec
// with complex(8) fields, modMLFMA.f90:1783-1946.)
//
// FP32 operator: radiation patterns, translation tables, interpolation and
// anterpolation weights, phase-shift tables and all C/B/A fields are float;
// every stage accumulates in FP32 on the CUDA cores, which GB300 runs 64x
// faster than FP64; the near field is the reference's complex(4) block
// itself.  Input and output vectors stay complex(8).
//
// Refinement (mode 1 of mlf_solve): r = b - A64 x in FP64; one restart cycle
// of right-preconditioned GMRES(m) solves A d = r with an FP32 inner loop
// (operator, preconditioner, Krylov basis and Gram-Schmidt in float) until its
// residual estimate drops below inner_tol ||b|| or m steps; x += M^-1 V y,
// accumulated in FP64; stop when the FP64 residual ||b - A64 x|| < tol ||b||.
// The FP64 residual decides, so the result meets the same stopping test as
// the plain FP64 solve.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <memory>
#include <type_traits>
#include <vector>

#include "mlf_cvt.cuh"
#include "mlf_f32x2.cuh"
#include "mlf_internal.h"
#include "mlf_sep.cuh"

namespace mlf {

#define CK(call)                                             \
    do {                                                     \
        if (!cuda_ok(c, (call), #call)) return MLF_E_CUDA;   \
    } while (0)

__device__ __forceinline__ void fmac(float2& acc, float2 a, float2 b) {
    acc.x = fmaf(a.x, b.x, acc.x);
    acc.x = fmaf(-a.y, b.y, acc.x);
    acc.y = fmaf(a.x, b.y, acc.y);
    acc.y = fmaf(a.y, b.x, acc.y);
}

// Krylov basis storage: FP32, or FP16 scaled by s = sqrt(N) on store (a unit
// column has every entry within sqrt(N), inside FP16's range) and by 1/s on
// load.  Arithmetic stays FP32 either way.
__device__ __forceinline__ float2 bload(const float2* p, float) { return *p; }
__device__ __forceinline__ float2 bload(const __half2* p, float s) {
    const float2 v = __half22float2(*p);
    return make_float2(v.x * s, v.y * s);
}
__device__ __forceinline__ void bstore(float2* p, float2 v, float) { *p = v; }
__device__ __forceinline__ void bstore(__half2* p, float2 v, float s) { *p = __floats2half2_rn(v.x * s, v.y * s); }

__global__ void k32_from64(size_t n, const double2* __restrict__ a, float2* __restrict__ b) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        b[i] = make_float2(d2f(a[i].x), d2f(a[i].y));
}

// x (FP64, ld) -> packed FP32 columns
__global__ void k32_pack_x(int N, int nrhs, int ld, const double2* __restrict__ x, float2* __restrict__ xf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    if (i < N) {
        const double2 v = x[(size_t)r * ld + i];
        xf[(size_t)r * N + i] = make_float2(d2f(v.x), d2f(v.y));
    }
}

__global__ void k32_aggregate(int K, int nrhs, int N, const int* __restrict__ box_ptr, const int* __restrict__ perm,
                              const float2* __restrict__ R, const float2* __restrict__ xf, float2* __restrict__ C) {
    const int b = blockIdx.x / nrhs, r = blockIdx.x % nrhs;
    const int j0 = box_ptr[b], j1 = box_ptr[b + 1];
    const float2* xr = xf + (size_t)r * N;
    for (int q = threadIdx.x; q < 2 * K; q += blockDim.x) {
        float2 acc = make_float2(0.f, 0.f);
        for (int j = j0; j < j1; ++j) fmac(acc, R[(size_t)j * 2 * K + q], xr[perm[j]]);
        C[((size_t)b * nrhs + r) * 2 * K + q] = acc;
    }
}

// 16 bytes if on, else r as it was (not read then): the load is predicated, so
// that it can be issued ahead of the branch that uses it
__device__ __forceinline__ void ldg128_if(bool on, float4& r, const float4* p) {
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t@q ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "+f"(r.x), "+f"(r.y), "+f"(r.z), "+f"(r.w)
        : "l"(p), "r"((unsigned)on));
}

// B(:, col, box) = wq * sum over the far boxes of T_tid * C(:, col, src)
// (llenar_campoCyB, modMLFMA.f90:1838-1852), for a group of G consecutive boxes
// (G i .. G i + G - 1, in depth-first order and mostly siblings) over the
// merged list of their far boxes: each source value read serves every box of
// the group that has it.  A thread owns two consecutive samples (K = 2 L^2 is
// even), both polarisations, NR columns and the G boxes, in registers: 16-byte
// loads, and the index, address and branch work of a source is spent once for
// 4 NR values.  The sums C Re T and C Im T are kept apart, (Re, Im) of C in one
// packed FMA each, and joined at the end: no value is swapped or negated.
// One warp per CTA: what bounds the stage is the reads through L1 and L2 (44 GB
// of them on the sphere below), and groups in one CTA (2 to 8 warps, for L1
// hits) were up to 15 % slower, as were 4 boxes (3.5 ms), two and three sources
// in flight (3.0, 3.5 ms).  69120-RWG sphere, 16 columns: 2.97 -> 2.58 ms;
// 122880-RWG sphere, one column: 0.449 -> 0.389 ms; 30720-RWG spheroid, 64
// columns: 0.180 -> 0.141 ms (before: one sample a thread, unpacked, 4 boxes).
// The levels share a launch: a small one alone leaves SMs idle (the product
// of one column of 122880 unknowns 961 -> 846 us, of 30720 x 64 530 -> 521, of 69120 x
// 16 5614 -> 5530).
struct Tr32Level {
    int KP, nb, nchunk;
    unsigned block0;                  // first of its (group, chunk) blocks
    const int *gptr, *gsrc, *gtid;
    const float4* T;
    const float2* wq;
    const float4* C;
    float4* B;
};
constexpr int TR32_LEVELS = 16;       // levels of one launch
struct Tr32Levels {
    Tr32Level l[TR32_LEVELS];
    int n;
};

template <int NR, int G>
__global__ void __launch_bounds__(32) k32_translate_grp(int nrhs, const __grid_constant__ Tr32Levels ls) {
    int lv = 0;
    while (lv + 1 < ls.n && blockIdx.x >= ls.l[lv + 1].block0) ++lv;
    const Tr32Level& l = ls.l[lv];
    const int KP = l.KP, nb = l.nb, nchunk = l.nchunk, bx = (int)(blockIdx.x - l.block0);
    const int *__restrict__ gptr = l.gptr, *__restrict__ gsrc = l.gsrc, *__restrict__ gtid = l.gtid;
    const float4 *__restrict__ T = l.T, *__restrict__ C = l.C;
    const float2* __restrict__ wq = l.wq;
    float4* __restrict__ B = l.B;
    const int gr = bx / nchunk;
    const int c0 = blockIdx.y * NR;
    const int k = bx % nchunk * 32 + threadIdx.x;   // pair of samples
    if (k >= KP) return;
    f32x2 a[G][2 * NR][2], b[G][2 * NR][2];   // sums of C Re T and C Im T, per box, slot and sample
#pragma unroll
    for (int h = 0; h < G; ++h)
#pragma unroll
        for (int u = 0; u < 2 * NR; ++u) a[h][u][0] = a[h][u][1] = b[h][u][0] = b[h][u][1] = 0;
    const float4* Cu[2 * NR];   // columns past the last read the last one's values
#pragma unroll
    for (int u = 0; u < 2 * NR; ++u) Cu[u] = C + (size_t)(2 * min(c0 + u / 2, nrhs - 1) + u % 2) * KP + k;
    const size_t cstride = 2 * (size_t)nrhs * KP;
    const float4* Tk = T + k;
    const int e1 = gptr[gr + 1];
    for (int e = gptr[gr]; e < e1; ++e) {
        int t[G];   // the same for the whole warp: uniform branches
        const size_t so = (size_t)gsrc[e] * cstride;
        if (G == 4) {
            const int4 q = reinterpret_cast<const int4*>(gtid)[e];
            t[0] = q.x; t[1 % G] = q.y; t[2 % G] = q.z; t[3 % G] = q.w;
        } else if (G == 2) {
            const int2 q = reinterpret_cast<const int2*>(gtid)[e];
            t[0] = q.x; t[1 % G] = q.y;
        } else {
            t[0] = gtid[e];
        }
        float4 v[2 * NR], w[G];
#pragma unroll
        for (int u = 0; u < 2 * NR; ++u) v[u] = Cu[u][so];
#pragma unroll
        for (int h = 0; h < G; ++h) ldg128_if(t[h] >= 0, w[h], Tk + (size_t)t[h] * KP);
#pragma unroll
        for (int h = 0; h < G; ++h)
            if (t[h] >= 0) {
                const f32x2 x0 = pk2(w[h].x, w[h].x), y0 = pk2(w[h].y, w[h].y);
                const f32x2 x1 = pk2(w[h].z, w[h].z), y1 = pk2(w[h].w, w[h].w);
#pragma unroll
                for (int u = 0; u < 2 * NR; ++u) {
                    const f32x2 p0 = pk2(v[u].x, v[u].y), p1 = pk2(v[u].z, v[u].w);
                    a[h][u][0] = fma2(p0, x0, a[h][u][0]);
                    b[h][u][0] = fma2(p0, y0, b[h][u][0]);
                    a[h][u][1] = fma2(p1, x1, a[h][u][1]);
                    b[h][u][1] = fma2(p1, y1, b[h][u][1]);
                }
            }
    }
    const float2 wk = wq[k];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        const int box = G * gr + h;
        if (box >= nb) break;
#pragma unroll
        for (int u = 0; u < 2 * NR; ++u)
            if (c0 + u / 2 < nrhs) {
                const float2 a0 = up2(a[h][u][0]), b0 = up2(b[h][u][0]), a1 = up2(a[h][u][1]), b1 = up2(b[h][u][1]);
                B[((size_t)box * nrhs + c0) * 2 * KP + (size_t)u * KP + k] =
                    make_float4((a0.x - b0.y) * wk.x, (a0.y + b0.x) * wk.x, (a1.x - b1.y) * wk.y, (a1.y + b1.x) * wk.y);
            }
    }
}

// FP32 interpolation between octree levels (the separable upward pass of
// mlf_sep.cuh) for NS field slots (columns x polarisations of a box) a thread,
// with packed FMAs on (Re, Im).  Slots past the last read the last one's values.
//   Cp(ip, it) = sum over the children of shift * sum_b wph sum_a wth Cc
// blockIdx.x = (parent, slot group, slab of `rows` coarse theta rows); thread =
// coarse sample (ip, it), so its stencil indices and weights are loaded once for
// all children and slots; slabs are cut so that their samples fill a CTA of at
// most IN32_T threads.  Y (shared memory, two buffers, [fine phi][row] with the
// NS slots side by side, padded to NS + 2: no bank conflicts at 16 bytes) =
// theta pass of one child; the phi pass sums v Re(shift) and v Im(shift) over
// the children in registers.  Latency bounds it, so warps in flight count:
// four slots at 64 registers (1.06 ms on the 69120-RWG sphere, 16 columns)
// against eight (1.11) and CTAs of 384 (1.48); with 8-row slabs, 256 threads
// and the parent slab in shared memory it was 1.34 ms.  One column of the
// 122880-RWG sphere: 0.163 -> 0.141 ms.
constexpr int IN32_T = 256;
template <int NS>
__global__ void __launch_bounds__(IN32_T, NS == 2 ? 6 : 4)
k32_interp(int Lp, int Lc, int nslot, int nsg, int nslab, int rows, const int* __restrict__ child_ptr,
           const int* __restrict__ octant, const int* __restrict__ sth, const float* __restrict__ wth,
           const int* __restrict__ sph, const float* __restrict__ wph, const float2* __restrict__ shift,
           const float2* __restrict__ Cc, float2* __restrict__ Cp) {
    extern __shared__ __align__(16) unsigned char sep_smem[];
    constexpr int SS = NS + 2;   // float2 per intermediate sample
    float2* Y = reinterpret_cast<float2*>(sep_smem);
    const int slab = blockIdx.x % nslab, sg = blockIdx.x / nslab % nsg, P = blockIdx.x / nslab / nsg;
    const int q0 = sg * NS, i0 = slab * rows, nr = min(rows, Lp - i0);
    const int Kp = 2 * Lp * Lp, Kc = 2 * Lc * Lc;
    const int hi = threadIdx.x / nr, li = threadIdx.x - hi * nr;   // column (fine phi, then coarse phi), row
    const bool th_on = hi < 2 * Lc, ph_on = hi < 2 * Lp;
    int fa[3] = {0, 0, 0}, fb[3] = {0, 0, 0};
    f32x2 wa[3], wb[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        float w = 0.f;
        if (th_on) { w = wth[3 * (i0 + li) + t]; fa[t] = sth[3 * (i0 + li) + t] + hi * Lc; }
        wa[t] = pk2(w, w);
        w = 0.f;
        if (ph_on) { w = wph[3 * hi + t]; fb[t] = (sph[3 * hi + t] * rows + li) * SS; }
        wb[t] = pk2(w, w);
    }
    const int ks = hi * Lp + i0 + li;   // coarse sample
    f32x2 sr[NS], si[NS];
#pragma unroll
    for (int u = 0; u < NS; ++u) sr[u] = si[u] = 0;
    const int c0 = child_ptr[P], c1 = child_ptr[P + 1], nbuf = 2 * Lc * rows * SS;
    for (int cb = c0; cb < c1; ++cb) {
        float2* Yb = Y + ((cb - c0) & 1) * nbuf;
        if (th_on) {
            const float2* src = Cc + ((size_t)cb * nslot + q0) * Kc;
            f32x2 y[NS];
#pragma unroll
            for (int u = 0; u < NS; ++u) {
                const float2* col = src + (size_t)min(u, nslot - 1 - q0) * Kc;
                y[u] = 0;
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const float2 v = col[fa[t]];
                    y[u] = fma2(pk2(v.x, v.y), wa[t], y[u]);
                }
            }
            float4* d = reinterpret_cast<float4*>(Yb + (hi * rows + li) * SS);
#pragma unroll
            for (int u = 0; u < NS; u += 2) {
                const float2 v0 = up2(y[u]), v1 = up2(y[u + 1]);
                d[u / 2] = make_float4(v0.x, v0.y, v1.x, v1.y);
            }
        }
        __syncthreads();   // two buffers: one barrier a child
        if (ph_on) {
            const float2 z = shift[(size_t)octant[cb] * Kp + ks];
            const f32x2 zr = pk2(z.x, z.x), zi = pk2(z.y, z.y);
            f32x2 v[NS];
#pragma unroll
            for (int u = 0; u < NS; ++u) v[u] = 0;
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const float4* yq = reinterpret_cast<const float4*>(Yb + fb[t]);
#pragma unroll
                for (int u = 0; u < NS; u += 2) {
                    const float4 q = yq[u / 2];
                    v[u] = fma2(pk2(q.x, q.y), wb[t], v[u]);
                    v[u + 1] = fma2(pk2(q.z, q.w), wb[t], v[u + 1]);
                }
            }
#pragma unroll
            for (int u = 0; u < NS; ++u) {
                sr[u] = fma2(v[u], zr, sr[u]);
                si[u] = fma2(v[u], zi, si[u]);
            }
        }
    }
    if (ph_on) {
        float2* dst = Cp + ((size_t)P * nslot + q0) * Kp + ks;
#pragma unroll
        for (int u = 0; u < NS; ++u)
            if (q0 + u < nslot) {
                const float2 a = up2(sr[u]), b = up2(si[u]);
                dst[(size_t)u * Kp] = make_float2(a.x - b.y, a.y + b.x);
            }
    }
}

__global__ void k32_receive_near(int K, int N, int nrhs, int ld, const int* __restrict__ perm,
                                 const int* __restrict__ box_of_sorted, const float2* __restrict__ R,
                                 const float2* __restrict__ A, const int* __restrict__ ia, const int* __restrict__ ja,
                                 const float2* __restrict__ Z, const float2* __restrict__ xf, float facy,
                                 double2* __restrict__ y) {
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (gw >= N * nrhs) return;
    const int j = gw / nrhs, r = gw % nrhs;
    const int n = perm[j], b = box_of_sorted[j];
    const float2* Rj = R + (size_t)j * 2 * K;
    const float2* Ab = A + ((size_t)b * nrhs + r) * 2 * K;
    float sr = 0.f, si = 0.f;
    for (int q = lane; q < 2 * K; q += 32) {
        const float2 a = Rj[q], v = Ab[q];
        sr = fmaf(a.x, v.x, sr); sr = fmaf(a.y, v.y, sr);
        si = fmaf(a.x, v.y, si); si = fmaf(-a.y, v.x, si);
    }
    const float2* xr = xf + (size_t)r * N;
    float nr = 0.f, ni = 0.f;
    for (int q = ia[n] + lane; q < ia[n + 1]; q += 32) {
        const float2 z = Z[q];
        const float2 xv = xr[ja[q]];
        nr = fmaf(xv.x, z.x, nr); nr = fmaf(-xv.y, z.y, nr);
        ni = fmaf(xv.x, z.y, ni); ni = fmaf(xv.y, z.x, ni);
    }
    float tr = fmaf(-facy, si, nr), ti = fmaf(facy, sr, ni);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        tr += __shfl_xor_sync(0xffffffff, tr, o);
        ti += __shfl_xor_sync(0xffffffff, ti, o);
    }
    if (lane == 0) y[(size_t)r * ld + n] = make_double2(f2d(tr), f2d(ti));
}

// ---------------------------------------------------------------------------

static int up32(Ctx* c, float** dst, const std::vector<double>& v) {
    std::vector<float> f(v.begin(), v.end());
    CK(cudaMalloc(dst, std::max<size_t>(f.size(), 1) * sizeof(float)));
    if (!f.empty()) CK(cudaMemcpy(*dst, f.data(), f.size() * sizeof(float), cudaMemcpyHostToDevice));
    return MLF_OK;
}

static int conv32(Ctx* c, float2** dst, const double2* src, size_t n) {
    CK(cudaMalloc(dst, std::max<size_t>(n, 1) * sizeof(float2)));
    if (n) k32_from64<<<(unsigned)std::min<size_t>((n + 255) / 256, 65535), 256, 0, c->stream>>>(n, src, *dst);
    CK(cudaGetLastError());
    return MLF_OK;
}

// Merged far lists of the box groups (G i .. G i + G - 1) of one level,
// sources ascending, with each source's translation index per box (-1 where
// it is not far from that box).
static int group_lists(Ctx* c, const Level& L, int G, Mixed32::Lv::Grp& M) {
    const int ng = (L.nb + G - 1) / G;
    std::vector<int> gptr(ng + 1, 0), gsrc, gtid;
    std::vector<std::pair<int, int>> ent;   // (source, box within the group), then the translation
    std::vector<int> etid;
    for (int g = 0; g < ng; ++g) {
        ent.clear();
        etid.clear();
        for (int h = 0; h < G && G * g + h < L.nb; ++h) {
            const int b = G * g + h;
            for (int f = L.far_ptr[b]; f < L.far_ptr[b + 1]; ++f) ent.push_back({L.far_src[f], (h << 20) | (int)etid.size()}), etid.push_back(L.far_tid[f]);
        }
        std::sort(ent.begin(), ent.end());
        for (size_t q = 0; q < ent.size(); ++q) {
            const int h = ent[q].second >> 20, t = etid[ent[q].second & 0xfffff];
            if (q == 0 || ent[q].first != ent[q - 1].first) {
                gsrc.push_back(ent[q].first);
                gtid.insert(gtid.end(), G, -1);
            }
            gtid[gtid.size() - G + h] = t;
        }
        gptr[g + 1] = (int)gsrc.size();
    }
    for (int* p : {M.ptr, M.src, M.tid})   // of an attempt that failed
        if (p) cudaFree(p);
    M.ptr = M.src = M.tid = nullptr;
    CK(cudaMalloc(&M.src, std::max<size_t>(gsrc.size(), 1) * sizeof(int)));
    CK(cudaMalloc(&M.tid, std::max<size_t>(gtid.size(), 4) * sizeof(int)));
    if (!gsrc.empty()) {
        CK(cudaMemcpy(M.src, gsrc.data(), gsrc.size() * sizeof(int), cudaMemcpyHostToDevice));
        CK(cudaMemcpy(M.tid, gtid.data(), gtid.size() * sizeof(int), cudaMemcpyHostToDevice));
    }
    CK(cudaMalloc(&M.ptr, gptr.size() * sizeof(int)));   // last: a set pointer means complete lists
    CK(cudaMemcpy(M.ptr, gptr.data(), gptr.size() * sizeof(int), cudaMemcpyHostToDevice));
    return MLF_OK;
}

// lists for groups of 4 boxes, which only mlf_set_translation_group asks for
static int quad_lists(Ctx* c) {
    for (int n = 3; n <= c->nlev; ++n) {
        Mixed32::Lv::Grp& g = c->m32.lv[n].grp[1];
        if (g.ptr) continue;
        const int st = group_lists(c, c->lv[n], 4, g);
        if (st) return st;
    }
    return MLF_OK;
}

int mixed_setup(Ctx* c) {
    if (c->m32.ready) return MLF_OK;
    const int nl = c->nlev;
    int st;
    if ((st = conv32(c, &c->m32.R, c->dR, (size_t)c->N * 2 * c->lv[nl].K))) return st;
    for (int n = 3; n <= nl; ++n) {
        Level& L = c->lv[n];
        Mixed32::Lv& M = c->m32.lv[n];
        if ((st = conv32(c, &M.T, L.dT, (size_t)L.ntrans * L.K))) return st;
        if ((st = up32(c, &M.wq, L.wq))) return st;
        if ((st = group_lists(c, L, 2, M.grp[0]))) return st;
        if (n < nl) {
            if ((st = up32(c, &M.wth, L.wth))) return st;
            if ((st = up32(c, &M.wph, L.wph))) return st;
            if ((st = up32(c, &M.thT_w, L.thT_w))) return st;
            if ((st = up32(c, &M.phT_w, L.phT_w))) return st;
            std::vector<double2> sh(8 * (size_t)L.K);
            CK(cudaMemcpy(sh.data(), L.dshift, sh.size() * sizeof(double2), cudaMemcpyDeviceToHost));
            std::vector<float2> s32(sh.size());
            for (size_t i = 0; i < sh.size(); ++i) s32[i] = make_float2((float)sh[i].x, (float)sh[i].y);
            CK(cudaMalloc(&M.shift, s32.size() * sizeof(float2)));
            CK(cudaMemcpy(M.shift, s32.data(), s32.size() * sizeof(float2), cudaMemcpyHostToDevice));
        }
    }
    size_t mx2 = 0, mx3 = 0;
    for (int n = 3; n < nl; ++n) {
        mx2 = std::max(mx2, ((size_t)c->lv[n].K + (size_t)c->lv[n].L * 2 * c->lv[n + 1].L) * sizeof(float2));
        mx3 = std::max(mx3, (size_t)SEP_SLAB * 2 * (c->lv[n + 1].L + c->lv[n].L) * sizeof(float2));
    }
    int optin = 0;
    CK(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->dev));
    if (mx2 > (size_t)optin || mx3 > (size_t)optin) {
        c->err = "parent sampling grid too large for the shared-memory interpolation stages";
        return MLF_E_ARG;
    }
    // kernel-wide limit shared by all contexts: the device maximum (see configure_kernels)
    CK(cudaFuncSetAttribute(k_anterp_sep<float2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    CK(cudaFuncSetAttribute(k_interp_sep<float2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    CK(cudaFuncSetAttribute(k32_interp<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    CK(cudaFuncSetAttribute(k32_interp<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin));
    if (c->tr_group == 4 && (st = quad_lists(c))) return st;
    CK(cudaStreamSynchronize(c->stream));
    c->m32.ready = 1;
    return MLF_OK;
}

static int ensure_fields32(Ctx* c, int nrhs) {
    if (c->m32.fcap >= nrhs && c->m32.xf) return MLF_OK;
    for (int n = 3; n <= c->nlev; ++n) {
        Mixed32::Lv& M = c->m32.lv[n];
        if (M.C) cudaFree(M.C);
        if (M.B) cudaFree(M.B);
        if (M.A) cudaFree(M.A);
        const size_t f = (size_t)c->lv[n].nb * nrhs * 2 * c->lv[n].K;
        CK(cudaMalloc(&M.C, f * sizeof(float2)));
        CK(cudaMalloc(&M.B, f * sizeof(float2)));
        CK(cudaMalloc(&M.A, f * sizeof(float2)));
    }
    if (c->m32.xf) cudaFree(c->m32.xf);
    CK(cudaMalloc(&c->m32.xf, (size_t)c->N * nrhs * sizeof(float2)));
    if (c->m32.xT) cudaFree(c->m32.xT);
    CK(cudaMalloc(&c->m32.xT, (size_t)c->N * nrhs * sizeof(float2)));
    c->m32.fcap = nrhs;
    return MLF_OK;
}

static int matvec32_core(Ctx* c, const double2* x, const float2* x32, double2* y, int nrhs, int ld, cudaStream_t s);

int device_matvec32(Ctx* c, const double2* x, double2* y, int nrhs, int ld, cudaStream_t s) {
    return matvec32_core(c, x, nullptr, y, nrhs, ld, s);
}

// y (FP64 columns, ld = N) = A32 x32 (FP32 packed columns)
int device_matvec32_from32(Ctx* c, const float2* x32, double2* y, int nrhs, cudaStream_t s) {
    return matvec32_core(c, nullptr, x32, y, nrhs, c->N, s);
}

// Field slots (columns x polarisations) per CTA of the anterpolation: the
// largest of 8, 4, 2 that divides 2 nrhs and keeps the CTA within 48 KB of
// shared memory (four CTAs per SM), else 1.  The slots share every index and
// weight load of the stencils.
template <class F>
static void slots_dispatch(int nrhs, size_t per_slot, F f) {
    const size_t cap = 48 * 1024;
    if ((2 * nrhs) % 8 == 0 && 8 * per_slot <= cap) f(std::integral_constant<int, 8>());
    else if ((2 * nrhs) % 4 == 0 && 4 * per_slot <= cap) f(std::integral_constant<int, 4>());
    else if (2 * per_slot <= cap) f(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, 1>());
}

static int matvec32_core(Ctx* c, const double2* x, const float2* x32, double2* y, int nrhs, int ld, cudaStream_t s) {
    int st;
    if (need_tree(c)) return MLF_E_STATE;
    if ((st = mixed_setup(c))) return st;
    if ((st = ensure_fields32(c, nrhs))) return st;
    const int nl = c->nlev;
    Level& leaf = c->lv[nl];
    const bool prof = c->profiling != 0;
    if (prof) cudaEventRecord(c->ev[0], s);
    const float2* xf = x32 ? x32 : c->m32.xf;
    if (nrhs == 1) {
        if (!x32) k32_pack_x<<<dim3((c->N + 255) / 256, nrhs), 256, 0, s>>>(c->N, nrhs, ld, x, c->m32.xf);
        k32_aggregate<<<leaf.nb * nrhs, 256, 0, s>>>(leaf.K, nrhs, c->N, c->dbox_ptr, c->dperm, c->m32.R, xf,
                                                     c->m32.lv[nl].C);
    } else {
        // blocks of columns: box-sorted row-major copy, then per-box GEMMs
        // (or one warp per basis for small boxes)
        if ((st = device_blk_pack(c, x, x32, ld, nrhs, c->m32.xT, s))) return st;
        const int eng = blk_engine_of(c);
        st = warp_engine(eng) ? device_agg_warp32(c, c->m32.R, leaf.K, c->m32.xT, nrhs, c->m32.lv[nl].C, s)
             : eng == 4       ? device_agg_tc(c, c->m32.R, leaf.K, c->m32.xT, nrhs, c->m32.lv[nl].C, s)
                              : device_agg_blocks32(c, c->m32.R, leaf.K, c->m32.xT, nrhs, c->m32.lv[nl].C, s);
        if (st) return st;
    }
    if (prof) cudaEventRecord(c->ev[1], s);
    for (int n = nl; n >= 4; --n) {
        Level& Lc = c->lv[n];
        Level& Lp = c->lv[n - 1];
        const Mixed32::Lv &mp = c->m32.lv[n - 1], &mc = c->m32.lv[n];
        if (Lc.L <= Lp.L && 2 * Lp.L <= IN32_T) {
            // slabs of coarse theta rows whose samples fill the CTA
            const int most = IN32_T / (2 * Lp.L), nslab = (Lp.L + most - 1) / most, rows = (Lp.L + nslab - 1) / nslab;
            const int threads = (rows * 2 * Lp.L + 31) / 32 * 32;
            auto launch = [&](auto ns) {
                constexpr int NS = decltype(ns)::value;
                const int nsg = (2 * nrhs + NS - 1) / NS;
                const size_t smem = (size_t)2 * 2 * Lc.L * rows * (NS + 2) * sizeof(float2);
                k32_interp<NS><<<Lp.nb * nsg * nslab, threads, smem, s>>>(
                    Lp.L, Lc.L, 2 * nrhs, nsg, nslab, rows, Lp.dchild_ptr, Lc.doctant, Lp.dsth, mp.wth, Lp.dsph,
                    mp.wph, mp.shift, mc.C, mp.C);
            };
            if (nrhs == 1) launch(std::integral_constant<int, 2>());
            else launch(std::integral_constant<int, 4>());
            continue;
        }
        const int nslab = (Lp.L + SEP_SLAB - 1) / SEP_SLAB;
        const size_t smem = (size_t)SEP_SLAB * 2 * (Lc.L + Lp.L) * sizeof(float2);   // child rows + parent slab
        k_interp_sep<float2, 1><<<Lp.nb * 2 * nrhs * nslab, 256, smem, s>>>(
            Lp.L, Lc.L, nrhs, nslab, Lp.dchild_ptr, Lc.doctant, Lp.dsth, mp.wth, Lp.dsph, mp.wph, mp.shift, mc.C,
            mp.C);
    }
    if (prof) cudaEventRecord(c->ev[2], s);
    for (int n = nl; n >= 3;) {   // from the leaves, as many levels as a launch takes
        const int G = c->tr_group ? c->tr_group : 2;
        const int nr = std::min(nrhs <= 1 ? 1 : nrhs <= 2 ? 2 : 4, c->tr_cols ? c->tr_cols : 2);
        Tr32Levels ls{};
        unsigned blocks = 0;
        for (; n >= 3 && ls.n < TR32_LEVELS; --n) {
            Level& L = c->lv[n];
            const Mixed32::Lv& m = c->m32.lv[n];
            const int KP = L.K / 2, nch = (KP + 31) / 32;
            ls.l[ls.n++] = {KP, L.nb, nch, blocks, G == 1 ? L.dfar_ptr : m.grp[G / 4].ptr,
                            G == 1 ? L.dfar_src : m.grp[G / 4].src, G == 1 ? L.dfar_tid : m.grp[G / 4].tid,
                            reinterpret_cast<const float4*>(m.T), reinterpret_cast<const float2*>(m.wq),
                            reinterpret_cast<const float4*>(m.C), reinterpret_cast<float4*>(m.B)};
            blocks += (unsigned)((L.nb + G - 1) / G * nch);
        }
        const dim3 grid(blocks, (nrhs + nr - 1) / nr);
#define TGRP(NR_, G_) k32_translate_grp<NR_, G_><<<grid, 32, 0, s>>>(nrhs, ls)
#define TNR(G_)                                                       \
    do {                                                              \
        if (nr == 1) TGRP(1, G_);                                     \
        else if (nr == 2) TGRP(2, G_);                                \
        else TGRP(4, G_);                                             \
    } while (0)
        if (G == 4) TNR(4);
        else if (G == 2) TNR(2);
        else TNR(1);
#undef TNR
#undef TGRP
    }
    if (prof) cudaEventRecord(c->ev[3], s);
    for (int n = 4; n <= nl; ++n) {
        Level& Lc = c->lv[n];
        Level& Lp = c->lv[n - 1];
        const float2* Psrc = (n == 4) ? c->m32.lv[n - 1].B : c->m32.lv[n - 1].A;
        const size_t per = ((size_t)Lp.K + (size_t)Lp.L * 2 * Lc.L) * sizeof(float2);
        const Mixed32::Lv &mp = c->m32.lv[n - 1], &mc = c->m32.lv[n];
        slots_dispatch(nrhs, per, [&](auto ns) {
            constexpr int NS = decltype(ns)::value;
            k_anterp_sep<float2, NS><<<Lc.nb * (2 * nrhs / NS), 256, NS * per, s>>>(
                Lp.L, Lc.L, nrhs, Lc.dparent, Lc.doctant, Lp.dthT_ptr, Lp.dthT_row, mp.thT_w, Lp.dphT_ptr,
                Lp.dphT_row, mp.phT_w, mp.shift, Psrc, mc.B, mc.A);
        });
    }
    if (prof) cudaEventRecord(c->ev[4], s);
    {
        const long long warps = (long long)c->N * nrhs;
        const float facy = (float)(c->ph.w * MU / (4. * PI));
        if (nrhs == 1) {
            k32_receive_near<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, s>>>(
                leaf.K, c->N, nrhs, ld, c->dperm, c->dbox_of_sorted, c->m32.R, (nl == 3 ? c->m32.lv[nl].B : c->m32.lv[nl].A), c->dia, c->dja,
                c->dZ, xf, facy, y);
        } else if (warp_engine(blk_engine_of(c))) {
            if ((st = device_recv_near_warp32(c, c->m32.R, leaf.K, (nl == 3 ? c->m32.lv[nl].B : c->m32.lv[nl].A), facy,
                                              c->m32.xT, nrhs, ld, y, s)))
                return st;
        } else {
            const float2* Aleaf = nl == 3 ? c->m32.lv[nl].B : c->m32.lv[nl].A;
            if (blk_engine_of(c) == 4) {
                // the X operand was packed by the aggregation of this product
                if ((st = device_recv_tc(c, c->m32.R, leaf.K, Aleaf, facy, nrhs, s))) return st;
                st = device_near_tc(c, ld, nrhs, y, s);
            } else {
                if ((st = device_recv_blocks32(c, c->m32.R, leaf.K, Aleaf, facy, nrhs, ld, y, s))) return st;
                st = device_near_blocks32(c, c->m32.xT, ld, nrhs, y, s);
            }
            if (st) return st;
        }
    }
    if (prof) cudaEventRecord(c->ev[5], s);
    if (!cuda_ok(c, cudaGetLastError(), "matvec32")) return MLF_E_CUDA;
    if (prof) {
        CK(cudaEventSynchronize(c->ev[5]));
        for (int i = 0; i < 5; ++i) cudaEventElapsedTime(&c->stage_ms[i], c->ev[i], c->ev[i + 1]);
    }
    return MLF_OK;
}

void mixed_free(Ctx* c) {
    auto F = [](void* p) { if (p) cudaFree(p); };
    F(c->m32.R); F(c->m32.xf); F(c->m32.xT); F(c->mix_ws);
    c->mix_ws = nullptr;
    c->mix_ws_bytes = 0;
    for (int n = 0; n < 32; ++n) {
        Mixed32::Lv& M = c->m32.lv[n];
        F(M.T); F(M.wq); F(M.shift); F(M.C); F(M.B); F(M.A);
        F(M.wth); F(M.wph); F(M.thT_w); F(M.phT_w);
        for (auto& g : M.grp) { F(g.ptr); F(g.src); F(g.tid); }
    }
}

// ---------------------------------------------------------------------------
// GMRES-IR: FP64 iterative refinement, each step one right-preconditioned
// GMRES(m) cycle on the FP32 operator (classical Gram-Schmidt, one pass by
// default, two with mlf_set_gs_passes).
// The reference's CGS (kept as mode 0) is too erratic to tolerate an
// operator perturbed at the 1e-7 level; GMRES minimises the residual over
// the Krylov space and cannot diverge.
// ---------------------------------------------------------------------------

constexpr int GM_BLOCKS = 128;

__global__ void k_resid(size_t n, const double2* __restrict__ b, const double2* __restrict__ Ax,
                        double2* __restrict__ r) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        r[i] = make_double2(b[i].x - Ax[i].x, b[i].y - Ax[i].y);
}
__global__ void k_axpy1(size_t n, const double2* __restrict__ d, double2* __restrict__ x) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        x[i].x += d[i].x;
        x[i].y += d[i].y;
    }
}

// partial[(i*nrhs + col)*GM_BLOCKS + blk] = sum conj(V_i) w   (grid: GM_BLOCKS, nrhs, nvec)
// or, with V == nullptr, sum |w|^2 in the real part (nvec = 1).
__global__ void k_mdot(int N, int nrhs, const double2* __restrict__ V, size_t vstride, const double2* __restrict__ w,
                       double2* __restrict__ partial) {
    const int col = blockIdx.y, i = blockIdx.z;
    const double2* wc = w + (size_t)col * N;
    const double2* vc = V ? V + i * vstride + (size_t)col * N : nullptr;
    double sr = 0, si = 0;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x) {
        const double2 b = wc[e];
        if (vc) {
            const double2 a = vc[e];   // conj(a) * b
            sr = fma(a.x, b.x, sr); sr = fma(a.y, b.y, sr);
            si = fma(a.x, b.y, si); si = fma(-a.y, b.x, si);
        } else {
            sr = fma(b.x, b.x, sr); sr = fma(b.y, b.y, sr);
        }
    }
    __shared__ double rs[256], is[256];
    rs[threadIdx.x] = sr;
    is[threadIdx.x] = si;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) { rs[threadIdx.x] += rs[threadIdx.x + s]; is[threadIdx.x] += is[threadIdx.x + s]; }
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[((size_t)i * nrhs + col) * gridDim.x + blockIdx.x] = make_double2(rs[0], is[0]);
}

// out[k] = sum_b partial[k*GM_BLOCKS + b], a warp each: four in order a lane, then
// halves (one thread's chain of FP64 additions, 64 cycles each, took 15.6 us)
__global__ void __launch_bounds__(32) k_reduce_partials(const double2* __restrict__ partial, double2* __restrict__ out) {
    const double2* p = partial + (size_t)blockIdx.x * GM_BLOCKS;
    double2 s = make_double2(0, 0);
#pragma unroll
    for (int b = 0; b < GM_BLOCKS / 32; ++b) {
        const double2 v = p[32 * b + threadIdx.x];
        s.x += v.x;
        s.y += v.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// FP32 Arnoldi kernels: basis V32 and work vector w32 in float, per-thread
// sums in float, block and final reductions in double.

// partial[col * gridDim.x + block] = sum |w|^2 of NRM_E values a thread, squares in
// float, sums in double (float -> double by moves); with a value a thread on 128 CTAs
// a column, and the sums of 128 partials by one thread each, the norms of 17280 x 32
// took 27 us, 9.7 now with the scales
constexpr int NRM_E = 8;
__global__ void __launch_bounds__(256) k_norm32(int N, const float2* __restrict__ w, double* __restrict__ partial) {
    const float2* wc = w + (size_t)blockIdx.y * N;
    double s = 0;
#pragma unroll
    for (int u = 0; u < NRM_E; ++u) {
        const int e = (blockIdx.x * NRM_E + u) * 256 + threadIdx.x;
        if (e < N) {
            const float2 v = wc[e];
            s += f2d(fmaf(v.y, v.y, v.x * v.x));
        }
    }
    __shared__ double ws[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 8; ++q) s += ws[q];
        partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = s;
    }
}

// norm[col].x = ||w(:, col)||^2, and scale[col], 1 or 0 for a column that runs or
// not, becomes 1 / ||w(:, col)|| (0 where that vanishes); a warp each
__global__ void __launch_bounds__(32) k_norm_scale(int nblk, const double* __restrict__ partial,
                                                   double2* __restrict__ norm, double* __restrict__ scale) {
    const int col = blockIdx.x;
    double s = 0;
    for (int b = threadIdx.x; b < nblk; b += 32) s += partial[(size_t)col * nblk + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x) return;
    norm[col] = make_double2(s, 0.0);
    const double h = sqrt(s);
    scale[col] = scale[col] != 0.0 && h > 1e-300 ? 1.0 / h : 0.0;
}

// Block dot products for the FP32 Arnoldi step: each CTA keeps its slice of
// w (MD_E values per thread) in registers and streams its share of the nvec
// basis vectors past it (blockIdx.z of gridDim.z shares, so that one column
// of 10^5 unknowns still fills the GPU), MD_G vectors per block reduction.
// partial[(i * nrhs + col) * gridDim.x + blockIdx.x] = sum conj(V_i) w over the slice.
constexpr int MD_E = 8, MD_G = 4;
template <class BT>
__global__ void __launch_bounds__(256) k_mdot32b(int N, int nrhs, int nvec, const BT* __restrict__ V,
                                                 size_t vstride, float ls, const float2* __restrict__ w,
                                                 double2* __restrict__ partial) {
    const int col = blockIdx.y;
    const size_t base = (size_t)col * N;
    const int e0 = blockIdx.x * 256 * MD_E + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ float red[8][2 * MD_G];
    float2 wv[MD_E];
#pragma unroll
    for (int u = 0; u < MD_E; ++u) {
        const int e = e0 + u * 256;
        wv[u] = e < N ? w[base + e] : make_float2(0.f, 0.f);
    }
    const int vper = ((nvec + gridDim.z - 1) / gridDim.z + MD_G - 1) / MD_G * MD_G;
    const int iend = min(nvec, (int)(blockIdx.z + 1) * vper);
    for (int i0 = blockIdx.z * vper; i0 < iend; i0 += MD_G) {
        float sacc[2 * MD_G];
#pragma unroll
        for (int g = 0; g < MD_G; ++g) {
            float sr = 0.f, si = 0.f;
            const int i = i0 + g;
            if (i < iend) {
                const BT* v = V + (size_t)i * vstride + base;
#pragma unroll
                for (int u = 0; u < MD_E; ++u) {
                    const int e = e0 + u * 256;
                    if (e < N) {
                        const float2 a = bload(v + e, ls);
                        sr = fmaf(a.x, wv[u].x, sr); sr = fmaf(a.y, wv[u].y, sr);
                        si = fmaf(a.x, wv[u].y, si); si = fmaf(-a.y, wv[u].x, si);
                    }
                }
            }
            sacc[2 * g] = sr;
            sacc[2 * g + 1] = si;
        }
        // warp sums of the 2 MD_G values by halving exchanges (MD_G = 4: 9
        // shuffles instead of 40): lane L ends with value (L >> 2)'s total
        static_assert(2 * MD_G == 8, "the exchange below is written for 8 values");
#pragma unroll
        for (int st = 0; st < 3; ++st) {
            const int o = 16 >> st, h = 4 >> st;
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q < h) {
                    const float send = up ? sacc[q] : sacc[q + h];
                    const float keep = up ? sacc[q + h] : sacc[q];
                    sacc[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
        }
        sacc[0] += __shfl_xor_sync(0xffffffffu, sacc[0], 2);
        sacc[0] += __shfl_xor_sync(0xffffffffu, sacc[0], 1);
        if ((lane & 3) == 0) red[warp][lane >> 2] = sacc[0];
        __syncthreads();
        if (threadIdx.x < MD_G && i0 + (int)threadIdx.x < iend) {
            double tr = 0, ti = 0;
            for (int wp = 0; wp < 8; ++wp) {
                tr += red[wp][2 * threadIdx.x];
                ti += red[wp][2 * threadIdx.x + 1];
            }
            partial[((size_t)(i0 + threadIdx.x) * nrhs + col) * gridDim.x + blockIdx.x] = make_double2(tr, ti);
        }
        __syncthreads();
    }
}

// out[k] = sum_b partial[k * nb + b], fixed order
__global__ void k_reduce_partials_n(int nk, int nb, const double2* __restrict__ partial, double2* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nk) return;
    double2 s = make_double2(0, 0);
#pragma unroll 16
    for (int b = 0; b < nb; ++b) {
        s.x += partial[(size_t)k * nb + b].x;
        s.y += partial[(size_t)k * nb + b].y;
    }
    out[k] = s;
}

template <class BT>
__global__ void k_gs_update32(int N, int nrhs, int nvec, const BT* __restrict__ V, size_t vstride, float ls,
                              const double2* __restrict__ h, float2* __restrict__ w) {
    const int col = blockIdx.y;
    __shared__ float2 hs[2048];
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
        const double2 hd = h[(size_t)i * nrhs + col];
        hs[i] = make_float2((float)hd.x, (float)hd.y);
    }
    __syncthreads();
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x) {
        float2 acc = w[(size_t)col * N + e];
        const BT* v = V + (size_t)col * N + e;
#pragma unroll 4
        for (int i = 0; i < nvec; ++i) {
            const float2 hv = hs[i];
            const float2 a = bload(v + (size_t)i * vstride, ls);
            acc.x -= hv.x * a.x - hv.y * a.y;
            acc.y -= hv.x * a.y + hv.y * a.x;
        }
        w[(size_t)col * N + e] = acc;
    }
}

template <class BT>
__global__ void k_colscale_df(int N, const double2* __restrict__ src, const double* __restrict__ s,
                              BT* __restrict__ dst, float ss) {
    const int col = blockIdx.y;
    const double f = s[col];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x) {
        const double2 v = src[(size_t)col * N + e];
        bstore(dst + (size_t)col * N + e, make_float2((float)(v.x * f), (float)(v.y * f)), ss);
    }
}

template <class BT>
__global__ void k_colscale32(int N, const float2* __restrict__ src, const double* __restrict__ s,
                             BT* __restrict__ dst, float ss) {
    const int col = blockIdx.y;
    const float f = (float)s[col];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x) {
        const float2 v = src[(size_t)col * N + e];
        bstore(dst + (size_t)col * N + e, make_float2(v.x * f, v.y * f), ss);
    }
}

// FP32 copy of one basis block (the preconditioner's input)
template <class BT>
__global__ void k_basis32(size_t n, const BT* __restrict__ src, float ls, float2* __restrict__ dst) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = bload(src + i, ls);
}

// d[col] = sum_i y[i*nrhs+col] V32_i[col] in double (once per cycle)
template <class BT>
__global__ void k_combine32(int N, int nrhs, int nvec, const BT* __restrict__ V, size_t vstride, float ls,
                            const double2* __restrict__ y, double2* __restrict__ d) {
    const int col = blockIdx.y;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N; e += gridDim.x * blockDim.x) {
        double2 acc = make_double2(0, 0);
        for (int i = 0; i < nvec; ++i) {
            const double2 yv = y[i * nrhs + col];
            const float2 v = bload(V + i * vstride + (size_t)col * N + e, ls);
            acc.x += yv.x * v.x - yv.y * v.y;
            acc.y += yv.x * v.y + yv.y * v.x;
        }
        d[(size_t)col * N + e] = acc;
    }
}

__global__ void k_d2f_m(size_t n, const double2* __restrict__ a, float2* __restrict__ b) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        b[i] = make_float2(d2f(a[i].x), d2f(a[i].y));
}
__global__ void k_f2d_m(size_t n, const float2* __restrict__ a, double2* __restrict__ b) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        b[i] = make_double2(f2d(a[i].x), f2d(a[i].y));
}

namespace {
struct Cx {
    double r, i;
};
inline Cx cx(double r, double i) { return {r, i}; }
inline Cx operator+(Cx a, Cx b) { return {a.r + b.r, a.i + b.i}; }
inline Cx operator-(Cx a, Cx b) { return {a.r - b.r, a.i - b.i}; }
inline Cx operator*(Cx a, Cx b) { return {a.r * b.r - a.i * b.i, a.r * b.i + a.i * b.r}; }
inline Cx conjx(Cx a) { return {a.r, -a.i}; }
inline double absx(Cx a) { return std::hypot(a.r, a.i); }
inline Cx divx(Cx a, Cx b) {
    const double d = b.r * b.r + b.i * b.i;
    return {(a.r * b.r + a.i * b.i) / d, (a.i * b.r - a.r * b.i) / d};
}
}  // namespace

static int col_norms(Ctx* c, int nrhs, const double2* w, double2* partial, double2* dred, std::vector<double2>& h,
                     std::vector<double>& out, cudaStream_t s) {
    k_mdot<<<dim3(GM_BLOCKS, nrhs, 1), 256, 0, s>>>(c->N, nrhs, nullptr, 0, w, partial);
    k_reduce_partials<<<nrhs, 32, 0, s>>>(partial, dred);
    CK(cudaMemcpyAsync(h.data(), dred, nrhs * sizeof(double2), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    for (int col = 0; col < nrhs; ++col) out[col] = std::sqrt(h[col].x);
    return MLF_OK;
}

static void col_norms32(int N, int nrhs, const float2* w, double2* partial, double2* norm, double* scale, cudaStream_t s) {
    const int nblk = (N + 256 * NRM_E - 1) / (256 * NRM_E);
    double* p = reinterpret_cast<double*>(partial);
    k_norm32<<<dim3(nblk, nrhs), 256, 0, s>>>(N, w, p);
    k_norm_scale<<<nrhs, 32, 0, s>>>(nblk, p, norm, scale);
}

// FP64 M^-1 applied to the correction once per cycle
static int apply_precond64(Ctx* c, int precond, int nrhs, const double2* in, double2* out, cudaStream_t s) {
    if (precond == 2) return device_nearinv_apply(c, in, out, nrhs, s);
    if (precond == 1) return device_ilu_solve(c, in, out, nrhs, s);
    CK(cudaMemcpyAsync(out, in, (size_t)c->N * nrhs * sizeof(double2), cudaMemcpyDeviceToDevice, s));
    return MLF_OK;
}

// Iterative refinement: r = b - A64 x (FP64); one cycle of right-preconditioned
// GMRES(m) with an all-FP32 inner loop (basis, Gram-Schmidt, preconditioner,
// operator; Hessenberg and Givens on the host in double); d = V y in double;
// x += M^-1 d (the neighbourhood inverse in FP32 as in the cycle, ILU0 in FP64).
// BT: the Krylov basis storage, float2 or __half2 (mlf_set_basis_precision).
template <class BT>
static int solve_mixed_t(Ctx* c, const double2* b, const double2* x0, double tol, int maxit, int nrhs, double2* x,
                         int* iters, double* relres, int precond, int* status, double inner_tol, int* outer) {
    const int N = c->N;
    // restart length: the one set, else 1600 while the basis fits in 16 GB,
    // down to 800 for wide blocks (a cold solve of the bench workloads takes
    // 1200-1600 steps; warm-started ones 500-800)
    const size_t colbytes = (size_t)N * nrhs * sizeof(BT);
    const int m_auto = (int)std::max<size_t>(800, std::min<size_t>(1600, ((size_t)16 << 30) / colbytes - 1));
    const int m = std::max(4, std::min(c->gmres_m > 0 ? c->gmres_m : m_auto, 2000));
    const size_t V1 = (size_t)N * nrhs;
    cudaStream_t s = c->stream;
    constexpr bool f32 = std::is_same<BT, float2>::value;
    const float ss = f32 ? 1.f : (float)std::sqrt((double)N), ls = 1.f / ss;   // store / load scales
    BT* V = nullptr;
    float2 *w32 = nullptr, *t32 = nullptr;
    double2 *w = nullptr, *r = nullptr, *t64 = nullptr, *partial = nullptr, *dred = nullptr;
    double* dscale = nullptr;
    const int md_chunks = (N + 256 * MD_E - 1) / (256 * MD_E);
    int nsm = 0;
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->dev));
    // The buffers come from a workspace the context keeps between solves: a
    // batched sweep solves hundreds of blocks, and allocating and freeing the
    // Krylov basis (tens of GB for wide blocks) for each took about 0.1 s.
    {
        auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
        const size_t sz[9] = {(size_t)(m + 1) * V1 * sizeof(BT), V1 * sizeof(float2), V1 * sizeof(float2),
                              V1 * sizeof(double2), V1 * sizeof(double2), V1 * sizeof(double2),
                              (size_t)(m + 1) * nrhs * std::max(GM_BLOCKS, md_chunks) * sizeof(double2),
                              (size_t)(m + 1) * nrhs * sizeof(double2), nrhs * sizeof(double)};
        size_t total = 0;
        for (size_t b : sz) total += al(b);
        if (c->mix_ws_bytes < total) {
            if (c->mix_ws) cudaFree(c->mix_ws);
            c->mix_ws = nullptr;
            c->mix_ws_bytes = 0;
            CK(cudaMalloc(&c->mix_ws, total));
            c->mix_ws_bytes = total;
        }
        char* p = static_cast<char*>(c->mix_ws);
        auto take = [&](int k) {
            char* q = p;
            p += al(sz[k]);
            return static_cast<void*>(q);
        };
        V = static_cast<BT*>(take(0));
        w32 = static_cast<float2*>(take(1));
        t32 = static_cast<float2*>(take(2));
        w = static_cast<double2*>(take(3));
        r = static_cast<double2*>(take(4));
        t64 = static_cast<double2*>(take(5));
        partial = static_cast<double2*>(take(6));
        dred = static_cast<double2*>(take(7));
        dscale = static_cast<double*>(take(8));
    }
    if (x0) CK(cudaMemcpyAsync(x, x0, V1 * sizeof(double2), cudaMemcpyDeviceToDevice, s));
    else CK(cudaMemsetAsync(x, 0, V1 * sizeof(double2), s));
    const unsigned g = (unsigned)std::min<size_t>((N + 255) / 256, 2048);
    const dim3 gc(g, nrhs);
    std::vector<double2> hbuf((size_t)(m + 1) * nrhs);
    std::vector<double> bn(nrhs), beta(nrhs), scl(nrhs);
    if (int st = col_norms(c, nrhs, b, partial, dred, hbuf, bn, s)) return st;
    std::fill(iters, iters + nrhs, 0);
    std::vector<int> done(nrhs, 0);
    // stagnation: the best FP64 residual of each column and the inner step count that reached it
    std::vector<double> sbest(nrhs, HUGE_VAL);
    std::vector<int> sbest_it(nrhs, 0);
    // H: per column the (m + 1) x m Hessenberg matrix, left uninitialised (for
    // wide blocks it spans hundreds of MB of which a cycle touches the first
    // few hundred columns): every entry is written before it is read
    std::unique_ptr<Cx[]> H(new Cx[(size_t)nrhs * (m + 1) * m]);
    std::vector<Cx> G((size_t)nrhs * (m + 1)), CS((size_t)nrhs * m), SN((size_t)nrhs * m);
    auto Hc = [&](int col, int i, int j) -> Cx& { return H[((size_t)col * m + j) * (m + 1) + i]; };
    int st = MLF_OK, k = 0;
    const int max_outer = 1000;
    const bool prof = c->profiling != 0;
    if (prof) {
        for (int q = 0; q < 4; ++q)
            if (!c->sev[q]) CK(cudaEventCreate(&c->sev[q]));
        for (double& v : c->solve_ms) v = 0;
    }
    const auto t_start = std::chrono::steady_clock::now();
    for (; k < max_outer; ++k) {
        // The residual that decides convergence is always FP64.  Two first
        // steps need no FP64 operator: with no initial guess r = b exactly;
        // with a warm start, the first cycle's right-hand side b - Z x0 is
        // formed with the FP32 operator and only feeds the inner solve (no
        // column is declared converged on it), the FP64 residual after the
        // cycle deciding as always.
        const bool provisional = k == 0 && x0 != nullptr;
        if (prof) cudaStreamSynchronize(s);
        const auto t_res = std::chrono::steady_clock::now();
        if (k == 0 && !x0) {
            CK(cudaMemcpyAsync(r, b, V1 * sizeof(double2), cudaMemcpyDeviceToDevice, s));
        } else {
            // after a check, only the columns still running need a new residual
            // (a converged column's x and r no longer change): they are gathered
            // so that the FP64 operator runs on those columns alone
            std::vector<int> run;
            if (!provisional)
                for (int col = 0; col < nrhs; ++col)
                    if (!done[col]) run.push_back(col);
            const int nrun = (int)run.size();
            c->mv_prec = provisional ? 1 : 0;
            if (!provisional && nrun < nrhs) {
                for (int i = 0; i < nrun && !st; ++i)
                    if (!cuda_ok(c, cudaMemcpyAsync(w + (size_t)i * N, x + (size_t)run[i] * N, N * sizeof(double2),
                                                    cudaMemcpyDeviceToDevice, s), "gather"))
                        st = MLF_E_CUDA;
                if (!st && nrun) st = device_matvec(c, w, t64, nrun, N, s);
                c->mv_prec = 0;
                if (st) break;
                for (int i = 0; i < nrun; ++i)
                    k_resid<<<1024, 256, 0, s>>>((size_t)N, b + (size_t)run[i] * N, t64 + (size_t)i * N,
                                                 r + (size_t)run[i] * N);
            } else {
                st = device_matvec(c, x, t64, nrhs, N, s);
                c->mv_prec = 0;
                if (st) break;
                k_resid<<<4096, 256, 0, s>>>(V1, b, t64, r);
            }
        }
        if ((st = col_norms(c, nrhs, r, partial, dred, hbuf, beta, s))) break;
        if (prof) {   // col_norms synchronised the stream
            const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_res).count();
            c->solve_ms[provisional ? 5 : 4] += ms;
        }
        bool all = true, budget = false;
        for (int col = 0; col < nrhs; ++col) {
            // a NaN or Inf in b or in the residual ends the column first
            // (bn > 0 is false for a NaN norm, which would read as converged)
            const bool finite = std::isfinite(bn[col]) && std::isfinite(beta[col]);
            relres[col] = !finite ? beta[col] / bn[col] : (bn[col] > 0 ? beta[col] / bn[col] : 0.0);
            if (!finite && !done[col]) { done[col] = 1; status[col] = MLF_CGS_NOT_FINITE; }
            if (!done[col] && !provisional && (relres[col] < tol || bn[col] == 0)) {
                done[col] = 1;
                status[col] = MLF_CGS_CONVERGED;
            }
            if (c->stag_window > 0 && !done[col] && !provisional) {
                if (relres[col] < sbest[col]) {
                    sbest[col] = relres[col];
                    sbest_it[col] = iters[col];
                } else if (iters[col] - sbest_it[col] >= c->stag_window) {
                    done[col] = 1;
                    status[col] = MLF_CGS_STAGNATED;
                }
            }
            all = all && done[col];
            budget = budget || (!done[col] && iters[col] < maxit);
        }
        if (all || !budget) break;
        for (int col = 0; col < nrhs; ++col) scl[col] = (!done[col] && beta[col] > 0) ? 1.0 / beta[col] : 0.0;
        CK(cudaMemcpyAsync(dscale, scl.data(), nrhs * sizeof(double), cudaMemcpyHostToDevice, s));
        k_colscale_df<BT><<<gc, 256, 0, s>>>(N, r, dscale, V, ss);
        std::fill(G.begin(), G.end(), cx(0, 0));
        for (int col = 0; col < nrhs; ++col) G[(size_t)col * (m + 1)] = cx(done[col] ? 0.0 : beta[col], 0);
        std::vector<int> jcol(nrhs, 0), live(nrhs, 0);
        for (int col = 0; col < nrhs; ++col) live[col] = !done[col];
        cudaGraphExec_t gexec = nullptr;
        for (int j = 0; j < m; ++j) {
            bool any = false;
            for (int col = 0; col < nrhs; ++col) any = any || live[col];
            if (!any) break;
            if (prof) cudaEventRecord(c->sev[0], s);
            for (int col = 0; col < nrhs; ++col) scl[col] = live[col] ? 1.0 : 0.0;   // for k_norm_scale
            CK(cudaMemcpyAsync(dscale, scl.data(), nrhs * sizeof(double), cudaMemcpyHostToDevice, s));
            const float2* vj;
            if (f32) {
                vj = reinterpret_cast<const float2*>(V + (size_t)j * V1);
            } else {   // w32 is free until the operator writes it below
                k_basis32<BT><<<4096, 256, 0, s>>>(V1, V + (size_t)j * V1, ls, w32);
                vj = w32;
            }
            if (precond == 2) {
                if ((st = device_nearinv_apply32(c, vj, t32, nrhs, s))) break;
            } else if (precond == 1) {
                k_f2d_m<<<4096, 256, 0, s>>>(V1, vj, w);
                if ((st = apply_precond64(c, 1, nrhs, w, t64, s))) break;
                k_d2f_m<<<4096, 256, 0, s>>>(V1, t64, t32);
            } else {
                CK(cudaMemcpyAsync(t32, vj, V1 * sizeof(float2), cudaMemcpyDeviceToDevice, s));
            }
            if (prof) cudaEventRecord(c->sev[1], s);
            // w32 = float(A32 t32): the first step of a cycle records these
            // launches (fixed buffers) into a CUDA graph, later steps replay it
            if (!gexec) {
                if ((st = device_matvec32_from32(c, t32, w, nrhs, s))) break;   // allocates lazily, uncaptured
                k_d2f_m<<<4096, 256, 0, s>>>(V1, w, w32);
                cudaGraph_t graph = nullptr;
                if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                    const int prof = c->profiling;
                    c->profiling = 0;
                    const int st2 = device_matvec32_from32(c, t32, w, nrhs, s);
                    k_d2f_m<<<4096, 256, 0, s>>>(V1, w, w32);
                    c->profiling = prof;
                    if (cudaStreamEndCapture(s, &graph) == cudaSuccess && st2 == MLF_OK && graph) {
                        if (cudaGraphInstantiate(&gexec, graph, 0) != cudaSuccess) gexec = nullptr;
                    }
                    if (graph) cudaGraphDestroy(graph);
                    cudaGetLastError();
                }
            } else {
                CK(cudaGraphLaunch(gexec, s));
            }
            if (prof) cudaEventRecord(c->sev[2], s);
            std::vector<double2> hsum((size_t)(j + 1) * nrhs, make_double2(0, 0));
            for (int pass = 0; pass < c->gs_passes; ++pass) {
                // vector shares when the slices alone leave SMs idle (under two CTAs
                // per SM): about four CTAs per SM in all, at least MD_G vectors each
                const int base_ctas = md_chunks * nrhs;
                const int vz = base_ctas >= 2 * nsm ? 1
                                                    : std::max(1, std::min((j + 1 + MD_G - 1) / MD_G,
                                                                           (4 * nsm + base_ctas - 1) / base_ctas));
                k_mdot32b<BT><<<dim3(md_chunks, nrhs, vz), 256, 0, s>>>(N, nrhs, j + 1, V, V1, ls, w32, partial);
                k_reduce_partials_n<<<((j + 1) * nrhs + 127) / 128, 128, 0, s>>>((j + 1) * nrhs, md_chunks, partial,
                                                                                  dred);
                k_gs_update32<BT><<<gc, 256, 0, s>>>(N, nrhs, j + 1, V, V1, ls, dred, w32);
                // the last pass's sums and the norms come back together, after the next
                // basis vector is on its way: one synchronisation a step
                const bool last = pass + 1 == c->gs_passes;
                if (last) {
                    col_norms32(N, nrhs, w32, partial, dred + (size_t)(j + 1) * nrhs, dscale, s);
                    k_colscale32<BT><<<gc, 256, 0, s>>>(N, w32, dscale, V + (size_t)(j + 1) * V1, ss);
                }
                CK(cudaMemcpyAsync(hbuf.data(), dred, (size_t)(j + 1 + last) * nrhs * sizeof(double2),
                                   cudaMemcpyDeviceToHost, s));
                CK(cudaStreamSynchronize(s));
                for (size_t q = 0; q < (size_t)(j + 1) * nrhs; ++q) { hsum[q].x += hbuf[q].x; hsum[q].y += hbuf[q].y; }
            }
            std::vector<double> hn(nrhs);
            for (int col = 0; col < nrhs; ++col) hn[col] = std::sqrt(hbuf[(size_t)(j + 1) * nrhs + col].x);
            if (prof) {
                cudaEventRecord(c->sev[3], s);
                cudaEventSynchronize(c->sev[3]);
                float a = 0, b2 = 0, d = 0;
                cudaEventElapsedTime(&a, c->sev[0], c->sev[1]);
                cudaEventElapsedTime(&b2, c->sev[1], c->sev[2]);
                cudaEventElapsedTime(&d, c->sev[2], c->sev[3]);
                c->solve_ms[0] += a; c->solve_ms[1] += b2; c->solve_ms[2] += d;
            }
            for (int col = 0; col < nrhs; ++col) {
                if (!live[col]) continue;
                for (int i = 0; i <= j; ++i) Hc(col, i, j) = cx(hsum[(size_t)i * nrhs + col].x, hsum[(size_t)i * nrhs + col].y);
                Hc(col, j + 1, j) = cx(hn[col], 0);
                for (int i = 0; i < j; ++i) {
                    const Cx a = Hc(col, i, j), bq = Hc(col, i + 1, j);
                    const Cx c_ = CS[(size_t)col * m + i], s_ = SN[(size_t)col * m + i];
                    Hc(col, i, j) = conjx(c_) * a + conjx(s_) * bq;
                    Hc(col, i + 1, j) = cx(0, 0) - s_ * a + c_ * bq;
                }
                const Cx a = Hc(col, j, j), bq = Hc(col, j + 1, j);
                const double nrm = std::hypot(absx(a), absx(bq));
                Cx c_ = cx(1, 0), s_ = cx(0, 0);
                if (nrm > 0) { c_ = divx(a, cx(nrm, 0)); s_ = divx(bq, cx(nrm, 0)); }
                CS[(size_t)col * m + j] = c_;
                SN[(size_t)col * m + j] = s_;
                Hc(col, j, j) = cx(nrm, 0);
                Hc(col, j + 1, j) = cx(0, 0);
                const Cx gj = G[(size_t)col * (m + 1) + j];
                G[(size_t)col * (m + 1) + j] = conjx(c_) * gj;
                G[(size_t)col * (m + 1) + j + 1] = cx(0, 0) - s_ * gj;
                jcol[col] = j + 1;
                iters[col] += 1;
                const double est = absx(G[(size_t)col * (m + 1) + j + 1]);
                if (est < inner_tol * bn[col] || hn[col] <= 1e-300 * bn[col] || iters[col] >= maxit) live[col] = 0;
            }
        }
        if (gexec) cudaGraphExecDestroy(gexec);
        if (st) break;
        std::vector<double2> y((size_t)(m + 1) * nrhs, make_double2(0, 0));
        int jmax = 0;
        for (int col = 0; col < nrhs; ++col) {
            const int jj = jcol[col];
            jmax = std::max(jmax, jj);
            std::vector<Cx> yy(jj);
            for (int i = jj - 1; i >= 0; --i) {
                Cx acc = G[(size_t)col * (m + 1) + i];
                for (int q = i + 1; q < jj; ++q) acc = acc - Hc(col, i, q) * yy[q];
                yy[i] = Hc(col, i, i).r != 0 || Hc(col, i, i).i != 0 ? divx(acc, Hc(col, i, i)) : cx(0, 0);
            }
            for (int i = 0; i < jj; ++i) y[(size_t)i * nrhs + col] = make_double2(yy[i].r, yy[i].i);
        }
        if (jmax == 0) break;
        CK(cudaMemcpyAsync(dred, y.data(), (size_t)jmax * nrhs * sizeof(double2), cudaMemcpyHostToDevice, s));
        k_combine32<BT><<<gc, 256, 0, s>>>(N, nrhs, jmax, V, V1, ls, dred, w);
        if (precond == 2 && f32) {
            // the correction through the FP32 neighbourhood inverse the cycle itself
            // used (the FP64 apply of a 64-column block costs ~0.12 s on GB300's
            // FP64 units; the FP32 one changes the correction by ~1e-6 relative,
            // and the FP64 residual still decides).  With the FP16 basis the FP64
            // apply stays: a 3-column solve on that basis then ran into its step
            // limit, which it meets with the FP64 apply.
            k_d2f_m<<<4096, 256, 0, s>>>(V1, w, w32);
            if ((st = device_nearinv_apply32(c, w32, t32, nrhs, s))) break;
            k_f2d_m<<<4096, 256, 0, s>>>(V1, t32, t64);
        } else if ((st = apply_precond64(c, precond, nrhs, w, t64, s))) {
            break;
        }
        k_axpy1<<<4096, 256, 0, s>>>(V1, t64, x);
        CK(cudaGetLastError());
    }
    c->mv_prec = 0;
    for (int col = 0; col < nrhs; ++col)
        if (!done[col]) status[col] = MLF_CGS_MAXIT;
    *outer = k;
    if (!st && blk_engine_of(c) == 4) st = tc_check(c);
    if (prof) {
        cudaStreamSynchronize(s);
        c->solve_ms[3] = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
        c->solve_ms[6] = k;
    }
    return st;
}

int device_solve_mixed(Ctx* c, const double2* b, const double2* x0, double tol, int maxit, int nrhs, double2* x,
                       int* iters, double* relres, int precond, int* status, double inner_tol, int* outer) {
    if (c->basis_bits == 16)
        return solve_mixed_t<__half2>(c, b, x0, tol, maxit, nrhs, x, iters, relres, precond, status, inner_tol, outer);
    return solve_mixed_t<float2>(c, b, x0, tol, maxit, nrhs, x, iters, relres, precond, status, inner_tol, outer);
}

}  // namespace mlf

using namespace mlf;

extern "C" int mlf_solve_times(mlf_ctx* h, double* out4) {
    if (!h || !out4) return MLF_E_ARG;
    for (int q = 0; q < 4; ++q) out4[q] = h->c.solve_ms[q];
    return MLF_OK;
}

extern "C" int mlf_solve_phases(mlf_ctx* h, double* out, int n) {
    if (!h || !out || n < 0) return MLF_E_ARG;
    for (int q = 0; q < n && q < 7; ++q) out[q] = h->c.solve_ms[q];
    return MLF_OK;
}

int mlf_set_gmres_restart(mlf_ctx* h, int m) {
    if (!h || (m != 0 && (m < 4 || m > 2000))) return MLF_E_ARG;
    h->c.gmres_m = m;
    return MLF_OK;
}

int mlf_set_gs_passes(mlf_ctx* h, int passes) {
    if (!h || passes < 1 || passes > 2) return MLF_E_ARG;
    h->c.gs_passes = passes;
    return MLF_OK;
}

int mlf_set_translation_group(mlf_ctx* h, int boxes, int cols) {
    if (!h || (boxes != 0 && boxes != 1 && boxes != 2 && boxes != 4) || (cols != 0 && cols != 1 && cols != 2 && cols != 4))
        return MLF_E_ARG;
    if (boxes == 4 && h->c.m32.ready) {   // before any product that a caller may capture
        Ctx* c = &h->c;
        if (!cuda_ok(c, cudaSetDevice(c->dev), "cudaSetDevice")) return MLF_E_CUDA;
        const int st = quad_lists(c);
        if (st) return st;
    }
    h->c.tr_group = boxes;
    h->c.tr_cols = cols;
    return MLF_OK;
}

int mlf_set_basis_precision(mlf_ctx* h, int bits) {
    if (!h || (bits != 16 && bits != 32)) return MLF_E_ARG;
    h->c.basis_bits = bits;
    return MLF_OK;
}

extern "C" int mlf_matvec32_device(mlf_ctx* h, const void* x, void* y, int nrhs, int ld, void* stream) {
    if (!h || !x || !y || nrhs <= 0 || ld < h->c.N) return MLF_E_ARG;
    Ctx* c = &h->c;
    if (!cuda_ok(c, cudaSetDevice(c->dev), "cudaSetDevice")) return MLF_E_CUDA;
    return device_matvec32(c, (const double2*)x, (double2*)y, nrhs, ld, stream ? (cudaStream_t)stream : c->stream);
}
