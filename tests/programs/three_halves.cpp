// Prints b, parm::three_halves(b) (parm_gb300/csrc/fpbits.cuh) as bit patterns
// for seeded values of b in (0, 1], of few bits, next to 1 and next to 0.  Test
// infrastructure.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "fpbits.cuh"

static uint64_t state = 0x9E3779B97F4A7C15ull;
static uint64_t next64() {   // splitmix64
    uint64_t z = (state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

static void show(double b) {
    const double r = parm::three_halves(b);
    uint64_t x, y;
    std::memcpy(&x, &b, 8);
    std::memcpy(&y, &r, 8);
    std::printf("%016llx %016llx\n", (unsigned long long)x, (unsigned long long)y);
}

int main() {
    for (int k = 0; k < 40000; k++) show((double)(next64() >> 11) * 0x1p-53);                    // 1 - R / sigma
    for (int k = 0; k < 20000; k++) show((double)(next64() >> 11) * 0x1p-53 * std::ldexp(1.0, -(k % 52)));
    for (int k = 1; k < 2000; k++) show(k * 0x1p-53), show(1.0 - k * 0x1p-53), show(k / 1024.0), show(k * k * 0x1p-53);
    show(0.0);
    show(1.0);
    show(2.0);
    return 0;
}
