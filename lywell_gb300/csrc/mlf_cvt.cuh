// FP32 <-> FP64 by moving the fields of the number.  A conversion instruction
// takes a slot of the FP64 pipe (a warp instruction in 19 cycles an SM, measured),
// which made kernels that only pass blocks on slower than memory; ordinary numbers
// and zeros take integer instructions here, the rest the instruction (volatile, so
// that it stays behind its branch).  Same bits as the conversions.
#pragma once

namespace mlf {

__device__ __forceinline__ double f2d(float f) {
    const unsigned u = __float_as_uint(f), ex = u >> 23 & 255u;
    if (ex - 1u < 254u || (u << 1) == 0)
        return __hiloint2double((int)((u & 0x80000000u) | ((u << 1) ? ((u & 0x7fffffffu) >> 3) + 0x38000000u : 0u)),
                                (int)(u << 29));
    double d;
    asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d) : "f"(f));
    return d;
}

__device__ __forceinline__ float d2f(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d), ex = hi >> 20 & 2047u;
    if (ex - 897u < 254u) {   // normal as FP32, or rounded up to infinity
        unsigned u = ((hi & 0x7fffffffu) - 0x38000000u) << 3 | lo >> 29;
        const unsigned r = lo & 0x1fffffffu;
        u += r > 0x10000000u || (r == 0x10000000u && (u & 1u));   // to nearest, ties to even
        return __uint_as_float(u | (hi & 0x80000000u));
    }
    if ((hi << 1 | lo) == 0) return __uint_as_float(hi);
    float f;
    asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(f) : "d"(d));
    return f;
}

}  // namespace mlf
