// Two short double-precision expressions of the reference, rounded to float,
// in float arithmetic alone: the back-projection quotient (W - 2 s) / (2 f)
// (transformation.cuh) and the blend's remaining transmittance
// rem (1 - w) (alphacompositing.cuh:58-68).
//
// Each is evaluated to about 2^-46 relative as a float r plus a correction:
// sums and products are split exactly into a rounded value and its error
// (T. J. Dekker, "A floating-point technique for extending the available
// precision", Numer. Math. 18, 1971).  The double expression differs from
// the exact value by a few 2^-53 relative, so as long as the estimate lies
// clearly within r's rounding interval, r is also what the double sequence
// rounds to.  Within 2^-16 of the interval's end (about one input in 2^15),
// and for operands outside the ranges checked below, the functions return
// false and the caller takes the exact integer path (uds_backproject.cuh,
// uds_blendrem.cuh) or the double arithmetic.  About 15 instructions each,
// against 100 to 200 for the integer paths.  The header also compiles as host
// C++ so that the CPU tests can compare it with the double formulas.
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define UDS_NF_FN __host__ __device__ __forceinline__
#else
#include <cmath>
#define UDS_NF_FN static inline
#endif

namespace uds {

#ifdef __CUDA_ARCH__
UDS_NF_FN float nf_add(float a, float b) { return __fadd_rn(a, b); }
UDS_NF_FN float nf_sub(float a, float b) { return __fsub_rn(a, b); }
UDS_NF_FN float nf_mul(float a, float b) { return __fmul_rn(a, b); }
UDS_NF_FN float nf_div(float a, float b) { return __fdiv_rn(a, b); }
UDS_NF_FN float nf_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
UDS_NF_FN uint32_t nf_bits(float x) { return __float_as_uint(x); }
UDS_NF_FN float nf_float(uint32_t u) { return __uint_as_float(u); }
#else
UDS_NF_FN float nf_add(float a, float b) { return a + b; }
UDS_NF_FN float nf_sub(float a, float b) { return a - b; }
UDS_NF_FN float nf_mul(float a, float b) { return a * b; }
UDS_NF_FN float nf_div(float a, float b) { return a / b; }
UDS_NF_FN float nf_fma(float a, float b, float c) { return fmaf(a, b, c); }
UDS_NF_FN uint32_t nf_bits(float x) {
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
}
UDS_NF_FN float nf_float(uint32_t u) {
    float x;
    memcpy(&x, &u, 4);
    return x;
}
#endif
UDS_NF_FN float nf_abs(float x) { return nf_float(nf_bits(x) & 0x7fffffffu); }

// Whether a value r + d (d to 2^-20 relative) lies clearly within the
// rounding interval of r: |d| below half a unit in the last place, a quarter
// where r is a power of two (the interval is shorter below it).  r must be
// at least 2^-100 in magnitude.
UDS_NF_FN bool nf_clear(float r, float d) {
    const uint32_t u = nf_bits(r) & 0x7fffffffu;
    const float half = nf_float((u & 0x7f800000u) - (24u << 23));
    return nf_abs(d) < ((u & 0x7fffffu) ? 0x1.fffep-1f : 0x1.fffep-2f) * half;
}

// (float)(((double)2 a - 2 s) / (2 f)); rf: 1 / f to 2^-22 relative
UDS_NF_FN bool near_quotient(float a, float s, float f, float rf, float* out) {
    const float hi = nf_sub(a, s);
    const float b = nf_sub(hi, a);
    const float lo = nf_sub(nf_sub(a, nf_sub(hi, b)), nf_add(s, b));  // a - s = hi + lo exactly
    const float q = nf_div(hi, f);
    const float aq = nf_abs(q), ah = nf_abs(hi);
    // magnitudes for which no error term underflows; NaNs fail here too
    if (!(f >= 0x1p-30f && f <= 0x1p30f && ah >= 0x1p-40f && ah <= 0x1p60f && aq >= 0x1p-60f)) return false;
    const float rest = nf_fma(-q, f, hi);  // exact
    const float c = nf_mul(nf_add(rest, lo), rf);
    const float r = nf_add(q, c);
    *out = r;
    return nf_clear(r, nf_add(nf_sub(q, r), c));
}

// (float)((double)rem * (1.0 - (double)w))
UDS_NF_FN bool near_rem(float rem, float w, float* out) {
    if (!(rem >= 0x1p-70f && rem <= 1.0f && w >= 0.0f && w <= 1.0f)) return false;
    const float hi = nf_sub(1.0f, w);
    const float lo = nf_sub(-w, nf_sub(hi, 1.0f));  // 1 - w = hi + lo exactly
    const float p = nf_mul(rem, hi);                // hi is 0 or at least 2^-24
    const float e = nf_fma(rem, hi, -p);            // exact
    const float t = nf_fma(rem, lo, e);
    const float r = nf_add(p, t);
    *out = r;
    return hi == 0.0f || nf_clear(r, nf_add(nf_sub(p, r), t));
}

}  // namespace uds
