// quotients.cuh -- the Q8_0 activation quantiser's divisions by multiplications, with the same bits.
// A block of 32 numbers v has d = RN(max|v| / 127) and the quants trunc(RN(v / d)) (buf_q8_0.rs:87-134); behind a norm v is RN(x / rms) * w.  Every CTA of a
// decode phase quantises the whole row for itself, and nine IEEE divisions for four numbers were most of that time (a 4096-row: 1.3 us of a phase of 15 to 20).
//   * a quotient by a divisor b that many numbers share: r = RN(1 / b) once, then two corrections q + (x - q b) r with fused multiply-adds.  The second starts
//     from a quotient within one unit in the last place, so it rounds correctly (P. Markstein, "Computation of elementary functions on the IBM RISC
//     System/6000 processor", 1990), as long as nothing underflows or overflows: cc_quot_range.
//   * trunc(RN(v / d)) for |v / d| <= 128: m = the whole number nearest to |v| * rcp, for a reciprocal within a few units; the remainder |v| - m d is exact (a
//     multiple of d's unit, small), and the rounded quotient reaches m if it is not below m by more than half a unit of the floats under m (a tie rounds to
//     m, whose mantissa is even).  Else the answer is m - 1.
// Plain C++ beside CUDA: the CPU test compiles this file.
#pragma once
#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define CC_QUOT_FN __host__ __device__ __forceinline__
#else
#define CC_QUOT_FN static inline
#endif

// magnitudes for which the corrections are exact, with room (0 is fine too)
CC_QUOT_FN bool cc_quot_range(float a) { return a >= 0x1p-60f && a <= 0x1p60f; }
CC_QUOT_FN float cc_quot_by(float x, float b, float r /* RN(1 / b) */) {
    float q = x * r;
    q = fmaf(fmaf(-b, q, x), r, q);
    return fmaf(fmaf(-b, q, x), r, q);
}
CC_QUOT_FN float cc_quot_float(int b) {
#ifdef __CUDA_ARCH__
    return __int_as_float(b);
#else
    float f; memcpy(&f, &b, 4); return f;
#endif
}
CC_QUOT_FN int cc_quot_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_int(f);
#else
    int b; memcpy(&b, &f, 4); return b;
#endif
}
// no non-zero number of the four below 2^-60 (doubled bits less one: zero becomes the largest)
CC_QUOT_FN bool cc_quot_no_tiny(float x, float y, float z, float w) {
    const unsigned a = ((unsigned)cc_quot_bits(x) << 1) - 1u, b = ((unsigned)cc_quot_bits(y) << 1) - 1u, c = ((unsigned)cc_quot_bits(z) << 1) - 1u, d = ((unsigned)cc_quot_bits(w) << 1) - 1u;
    const unsigned ab = a < b ? a : b, cd = c < d ? c : d;
    return (ab < cd ? ab : cd) >= (((127u - 60u) << 24) - 1u);
}
// d of a block
CC_QUOT_FN float cc_q8_0_scale(float amax) { return cc_quot_by(amax, 127.0f, 1.0f / 127.0f); }
// quant of v by d = RN(amax / 127), half = d / 2 and a reciprocal of d.  No number at all (NaN): 0, as the conversion of one
CC_QUOT_FN int cc_q8_0_quant(float v, float d, float half, float rcp) {
    const float a = fabsf(v);
    const float sh = a * rcp + 12582912.0f;                          // 1.5 * 2^23: the nearest whole number in the low bits
    const float m = sh - 12582912.0f;
    const float below = (cc_quot_float(cc_quot_bits(m) - 1) - m) * half;            // minus half a unit under m, times d (m = 0: NaN, nothing is below)
    int q = cc_quot_bits(sh) - 0x4B400000;
    if (fmaf(-m, d, a) < below) q--;
    const int sign = cc_quot_bits(v) >> 31;
    return (q ^ sign) - sign;
}
