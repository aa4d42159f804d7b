// quotients.cuh -- the Q8_0 activation quantiser's divisions by multiplications, with the same bits.
// A block of 32 numbers v has d = RN(max|v| / 127) and the quants trunc(RN(v / d)) (buf_q8_0.rs:87-134); behind a norm v is RN(x / rms) * w.  Every CTA of a
// decode phase quantises the whole row for itself, and nine IEEE divisions for four numbers were most of that time (a 4096-row: 1.3 us of a phase of 15 to 20).
//   * a quotient by a divisor b that many numbers share: r = RN(1 / b) once, then two corrections q + (x - q b) r with fused multiply-adds.  The second starts
//     from a quotient within one unit in the last place, so it rounds correctly (P. Markstein, "Computation of elementary functions on the IBM RISC
//     System/6000 processor", 1990), as long as nothing underflows or overflows: cc_quot_range.
//   * trunc(RN(v / d)): with any reciprocal within two units, v * rcp is within 127 * 2^-22 of the quotient, so its truncation is right unless a whole number lies
//     that close; then (and for the block's own maximum, whose quotient is 127 within a unit) the truth is worked out.
// Plain C++ beside CUDA: the CPU test compiles this file.
#pragma once
#include <math.h>

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
// d of a block, and the quant of its largest magnitude: amax / d is 127 or less than it by more than half of its unit 2^-17 (then 126)
CC_QUOT_FN float cc_q8_0_scale(float amax) { return cc_quot_by(amax, 127.0f, 1.0f / 127.0f); }
CC_QUOT_FN int cc_q8_0_top(float amax, float d) { return fmaf(d, 127.0f, -amax) > d * 0x1p-18f ? 126 : 127; }
// quant of v by a reciprocal of d; `doubt` is raised when a whole number is too close to tell
CC_QUOT_FN int cc_q8_0_quant(float v, float amax, int top, float rcp, bool& doubt) {
    const float t = v * rcp;
    const float whole = (t + 12582912.0f) - 12582912.0f;          // nearest whole number (|t| < 128)
    const bool is_top = fabsf(v) == amax;
    if (fabsf(t - whole) < 0x1p-14f && whole != 0.0f && !is_top) doubt = true;
#ifdef __CUDA_ARCH__
    const int q = __float2int_rz(t);
#else
    const int q = t == t ? (int)t : 0;
#endif
    return is_top ? (v < 0.0f ? -top : top) : q;
}
