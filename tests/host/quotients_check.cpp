// quotients.cuh on the CPU: prints the number of disagreements with IEEE division for each of its parts (tests/test_host_quotients.py).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

#include "../../crabml_b200/csrc/quotients.cuh"

static float from_bits(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t bits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }

int main() {
    long bad_scale = 0, bad_by = 0, bad_quant = 0, n_quant = 0, bad_tiny = 0;
    for (uint32_t m = 0; m < (1u << 23); m++)                                        // every mantissa, several exponents: the scale and the quant of the largest number
        for (uint32_t e : {68u, 127u, 128u, 186u}) {
            const float a = from_bits(e << 23 | m), d = a / 127.0f;
            if (bits(cc_q8_0_scale(a)) != bits(d)) bad_scale++;
            if (cc_q8_0_quant(e & 1 ? a : -a, d, 0.5f * d, 1.0f / d) != (e & 1 ? 1 : -1) * (int)(a / d)) bad_quant++;
        }
    std::mt19937 g(7);
    auto value = [&](int lo, int hi) { return from_bits((uint32_t)(127 + lo + (int)(g() % (uint32_t)(hi - lo))) << 23 | (g() & 0x7FFFFF) | (g() & 1u) << 31); };
    for (long i = 0; i < 60000000; i++) {                                            // shared divisors: random, and with mantissas at both ends
        float b = std::fabs(value(-20, 20));
        if (i % 3 == 1) b = from_bits((bits(b) & 0xFF800000u) | (g() % 64));
        if (i % 3 == 2) b = from_bits(bits(b) | (0x7FFFFF - g() % 64));
        const float x = i % 7 ? value(-50, 8) : b * (float)(g() % 4096) ;             // (and quotients that are nearly whole)
        if (x == 0.0f) continue;
        if (bits(cc_quot_by(x, b, 1.0f / b)) != bits(x / b)) bad_by++;
    }
    for (long i = 0; i < 3000000; i++) {                                             // blocks: random, and with quotients next to whole numbers
        const float amax = std::fabs(value(-50, 50)), d = amax / 127.0f;
        for (int wobble : {-2, -1, 0, 1, 2}) {                                       // a reciprocal that is off by up to two units
            const float rcp = from_bits(bits(1.0f / d) + wobble);
            float v = amax * (float)((int)(g() % 2000001) - 1000000) * 1e-6f;
            if (i % 2) v = from_bits(bits(d * (float)(g() % 127 + 1)) + (g() % 9) - 4) * (g() & 1 ? 1.0f : -1.0f);
            if (i % 5 == 0) v = wobble & 1 ? amax : -amax;
            if (std::fabs(v) > amax) continue;
            n_quant++;
            if (cc_q8_0_quant(v, d, 0.5f * d, rcp) != (int)(v / d)) bad_quant++;
        }
    }
    for (long i = 0; i < 1000000; i++) {
        float x[4]; bool tiny = false;
        for (float& f : x) { f = g() % 5 ? value(-64, -56) : 0.0f * (float)((int)(g() % 3) - 1); tiny = tiny || (f != 0.0f && std::fabs(f) < 0x1p-60f); }
        if (cc_quot_no_tiny(x[0], x[1], x[2], x[3]) == tiny) bad_tiny++;
    }
    printf("%ld %ld %ld %ld %ld\n", bad_scale, bad_by, bad_quant, bad_tiny, n_quant);
    return 0;
}
