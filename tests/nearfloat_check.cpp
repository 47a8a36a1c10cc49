// Host check of csrc/uds_nearfloat.cuh against the double formulas it
// replaces, bit for bit.  Prints, for each of the two, the number of inputs
// checked, how many the float path took, and mismatches.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "uds_nearfloat.cuh"

static unsigned long long s_state = 0x2545f4914f6cdd1dull;
static unsigned long long next64() {
    s_state ^= s_state << 13;
    s_state ^= s_state >> 7;
    s_state ^= s_state << 17;
    return s_state;
}
static float from_bits(unsigned u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
static unsigned to_bits(float f) {
    unsigned u;
    std::memcpy(&u, &f, 4);
    return u;
}
static float uniform01() { return (float)((next64() >> 40) * 0x1p-24); }
static float bit_uniform(float lo, float hi) {
    unsigned a = to_bits(lo), b = to_bits(hi);
    return from_bits(a + (unsigned)(next64() % (unsigned long long)(b - a + 1u)));
}

static long long n_rem = 0, fast_rem = 0, bad_rem = 0, n_q = 0, fast_q = 0, bad_q = 0;
static void rem(float r, float w) {
    ++n_rem;
    float got, ref = (float)((double)r * (1.0 - (double)w));
    if (uds::near_rem(r, w, &got)) {
        ++fast_rem;
        if (to_bits(got) != to_bits(ref) && bad_rem++ < 10) std::printf("rem %a %a: %a, not %a\n", r, w, got, ref);
    }
}
static void quotient(float W, float s, float f) {
    ++n_q;
    float got, ref = (float)(((double)W - 2.0 * (double)s) / (2.0 * (double)f));
    if (uds::near_quotient(W * 0.5f, s, f, 1.0f / f, &got)) {
        ++fast_q;
        if (to_bits(got) != to_bits(ref) && bad_q++ < 10)
            std::printf("quotient %a %a %a: %a, not %a\n", W, s, f, got, ref);
    }
}

int main(int argc, char** argv) {
    long long n = argc > 1 ? std::atoll(argv[1]) : 1000000;
    const float odd[] = {0.0f, -0.0f, 1.0f, 0.5f, 0x1p-24f, 0x1.fffffep-1f, 0x1.000002p+0f, 0x1p-70f, 0x1.fffffep-71f,
                         1e-38f, 1e-45f, 2.0f, -1.0f, 1e30f, from_bits(0x7f800000u), from_bits(0xff800000u),
                         from_bits(0x7fc00000u), 0x1p30f, 0x1p60f, 512.0f, 511.5f, 3.0f};
    for (float a : odd)
        for (float b : odd) {
            rem(a, b);
            for (float c : odd) quotient(a, b, c);
        }
    for (long long i = 0; i < n; ++i) {
        rem(uniform01(), uniform01());
        rem(bit_uniform(0x1p-72f, 1.0f), bit_uniform(0x1p-40f, 1.0f));
        rem(uniform01(), from_bits(0x3f800000u - (unsigned)(next64() % 4096u)));  // at and just below 1
        rem(uniform01(), (float)(next64() % 4097u) * 0x1p-12f);                   // products at rounding boundaries
        rem((float)(next64() % 4097u) * 0x1p-12f, uniform01());
        float W = (float)(1 + next64() % 4096u);
        quotient(W, (float)(next64() % 4096u), bit_uniform(0.25f, 8192.0f));       // pixels
        quotient(W, W * uniform01(), bit_uniform(0.25f, 8192.0f));
        quotient(W, W * 0.5f + bit_uniform(0x1p-30f, 2048.0f), W * uniform01() + 0.01f);
        quotient(W, (float)(next64() % 4096u) * 0.25f, (float)(1 + next64() % 512u));  // exact quotients, midpoints
        quotient(W, -bit_uniform(0x1p-20f, 0x1p20f), bit_uniform(0x1p-10f, 0x1p10f));
    }
    std::printf("%lld %lld %lld %lld %lld %lld\n", n_rem, fast_rem, bad_rem, n_q, fast_q, bad_q);
    return bad_rem || bad_q ? 1 : 0;
}
