// Checks parm::quotient_by_reciprocal (parm_gb300/csrc/fpbits.cuh) against the
// host's division on seeded random values of the range the force kernels use
// it in, on mantissas of few bits and on those next to them; prints
// "ok <count>" or the first mismatch.  Test infrastructure.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "fpbits.cuh"

static uint64_t sm_state = 0x9E3779B97F4A7C15ull;
static uint64_t next64() {   // splitmix64
    uint64_t z = (sm_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

static double make(uint64_t frac, int e) {
    const uint64_t b = ((uint64_t)(1023 + e) << 52) | (frac & 0xFFFFFFFFFFFFFull);
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}

static long count = 0;
static bool check(double a, double b) {
    count++;
    const double want = a / b, got = parm::quotient_by_reciprocal(a, b, 1 / b);
    if (std::memcmp(&want, &got, 8) == 0) return true;
    std::printf("mismatch: %.17g / %.17g -> %.17g, want %.17g\n", a, b, got, want);
    return false;
}

int main() {
    for (int k = 0; k < 20000000; k++) {
        const uint64_t r = next64();
        if (!check(make(next64(), (int)(r % 600) - 300), make(next64(), (int)((r >> 16) % 600) - 300))) return 1;
    }
    // mantissas at the ends and next to fractions of few bits
    for (uint64_t p = 0; p < 512; p++)
        for (int64_t dp = -3; dp <= 3; dp++)
            for (uint64_t q = 0; q < 512; q++)
                for (int64_t dq = -1; dq <= 1; dq++)
                    if (!check(make((p << 43) + (uint64_t)dp, 3), make((q << 43) + (uint64_t)dq, -1))) return 1;
    if (!check(0.0, 3.0) || !check(12.0, 1.0) || !check(-12.0, 7.0)) return 1;
    std::printf("ok %ld\n", count);
    return 0;
}
