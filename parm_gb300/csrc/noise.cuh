// Standard normals of the Langevin step: Philox4x32-10 (Salmon et al., SC'11)
// and Box-Muller, in FP64 with few FP64 operations.
//
// GB300 runs FP64 at 1/64 of its FP32 rate, and the library's log, sqrt and
// sincos take over a hundred FP64 operations per pair of normals, which bound
// the Langevin step.  Here the uniform variates stay integers until a table
// has taken out their leading bits (exact, integer instructions), the rest
// takes short polynomials whose high-order terms are FP32 (their rounding lies
// below an FP64 ulp of the sum), and the square root starts from the FP32
// reciprocal root: 33 FP64 operations per pair.
//   log:     P. T. P. Tang, "Table-driven implementation of the logarithm
//            function in IEEE floating-point arithmetic", ACM TOMS 16 (1990):
//            log(m 2^e) = e ln2 + log c + log1p(r), r = m / c - 1, the table's
//            last interval taken relative to c = 2 so that u near 1 keeps its
//            relative accuracy;
//   sin, cos: P. T. P. Tang, "Table-lookup algorithms for elementary functions
//            and their error analysis", ARITH-10 (1991): the angle's nearest
//            512th of a turn from the table, the rest by angle addition;
//   sqrt:    Newton's method on the reciprocal root with a final correction by
//            the exact remainder.
// Error in units of 2^-53 of the radius, against 113-bit arithmetic: at most 3.2,
// 0.58 rms over 1.2 million normals (log, sqrt and sincos of the library: 9.4 and
// 2.2, mostly the rounded angle).  48 WCA replicas of 256 to 32768 atoms,
// 16 steps with the records read back: 6.11 -> 4.54 ms.
#pragma once
#include <cmath>

#include "fpbits.cuh"

namespace parm {

constexpr uint32_t NOISE_LOG = 128, NOISE_TURN = 512;   // table sizes
struct NoiseTable {
    double lg[NOISE_LOG][2];    // 1 / c, -2 log c (less 2 ln2 for c > sqrt 2)
    double cs[NOISE_TURN][2];   // cos, sin of k / 512 turns
};
constexpr uint32_t NOISE_SPLIT = 53;   // first interval of [1, 2) above sqrt 2, taken with the next power of two

inline NoiseTable make_noise_table() {
    NoiseTable t;
    const long double ln2 = std::log(2.0L), turn = 2.0L * std::acos(-1.0L);
    for (uint32_t k = 0; k < NOISE_LOG; k++) {
        const long double mid = 1.0L + (2.0L * k + 1.0L) / (2.0L * NOISE_LOG);
        t.lg[k][0] = k == NOISE_LOG - 1 ? 0.5 : (double)(1.0L / mid);
        const long double lc = -std::log((long double)t.lg[k][0]) - (k >= NOISE_SPLIT ? ln2 : 0.0L);
        t.lg[k][1] = k == NOISE_LOG - 1 ? 0.0 : (double)(-2.0L * lc);
    }
    for (uint32_t k = 0; k < NOISE_TURN; k++) {
        // by octants, so that the exact values of the axes and diagonals are exact
        const uint32_t q = k / (NOISE_TURN / 4), r = k % (NOISE_TURN / 4);
        const bool fold = r > NOISE_TURN / 8;
        const long double a = turn * (fold ? NOISE_TURN / 4 - r : r) / NOISE_TURN;
        const double c0 = (double)(fold ? std::sin(a) : std::cos(a)), s0 = (double)(fold ? std::cos(a) : std::sin(a));
        t.cs[k][0] = q == 0 ? c0 : (q == 1 ? -s0 : (q == 2 ? -c0 : s0));
        t.cs[k][1] = q == 0 ? s0 : (q == 1 ? c0 : (q == 2 ? -s0 : -c0));
    }
    return t;
}

// the same constants for every handle, computed by the first that asks: where
// long double is done in software the ~400 logarithms, sines and cosines take
// 0.3 ms, a third of a new batch's first short call
inline const NoiseTable& noise_table() {
    static const NoiseTable t = make_noise_table();
    return t;
}

#if defined(__CUDACC__)
__device__ __forceinline__ void philox10(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
        uint32_t n0 = hi1 ^ c[1] ^ k0;
        uint32_t n2 = hi0 ^ c[3] ^ k1;
        c[0] = n0;
        c[1] = lo1;
        c[2] = n2;
        c[3] = lo0;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

// the 53-bit variate v of two words; the uniform in (0, 1] is (v + 1/2) 2^-53
__device__ __forceinline__ unsigned long long bits53(uint32_t a, uint32_t b) {
    return ((unsigned long long)(a >> 5) << 26) | (unsigned long long)(b >> 6);
}

// sqrt(-2 log u) of u = (v + 1/2) 2^-53 rounded to FP64
__device__ __forceinline__ double noise_radius(const NoiseTable* t, unsigned long long v) {
    // u 2^54 = 2 v + 1, rounded to 53 bits (ties to even) where it has 54
    unsigned long long w = 2ull * v + 1ull;
    if (v >> 52) w = (v + (v & 1ull)) << 1;
    const int lz = __clzll((long long)w);
    const unsigned long long frac = (w << lz) << 1;   // the leading 1 dropped, left-aligned
    const uint32_t k = (uint32_t)(frac >> 57);
    const int e = 9 - lz + (k >= NOISE_SPLIT ? 1 : 0);   // log2 of the leading bit - 54, + 1 above sqrt 2
    const double m = __hiloint2double((int)(0x3FF00000u | (uint32_t)(frac >> 44)), (int)(uint32_t)(frac >> 12));
    const double2 L = __ldg(reinterpret_cast<const double2*>(t->lg[k]));
    const double ed = f2d_flush((float)e);
    const double r = __fma_rn(m, L.x, -1.0);   // |r| < 2^-8
    // -2 log u = -2 ln2 e - 2 log c - 2 r + r^2 - 2/3 r^3 + ...; -2 ln2 in two parts, the first short enough
    // for an exact product with e
    constexpr double L2H = -0x1.62e42fefa38p+0, L2L = -0x1.ef35793c7673p-44;
    const double T = __fma_rn(ed, L2H, L.y);
    const double hi = __fma_rn(r, -2.0, T);
    double lo = __fma_rn(r, -2.0, __dsub_rn(T, hi));
    lo = __fma_rn(ed, L2L, lo);
    const float rf = d2f_chop(r);
    // r^5 to r^7, below 2^-33 of the sum; without r^7 the radius of u just above 255 / 256, where r is -2^-8 and the
    // first term is all there is beside it, was off by 2.8 units
    const float tail = rf * fmaf(rf, fmaf(rf, -2.0f / 7.0f, 1.0f / 3.0f), -0.4f);
    const double P = __fma_rn(r, __fma_rn(r, __dadd_rn(f2d_flush(tail), 0.5), -2.0 / 3.0), 1.0);
    double x = __dadd_rn(hi, __fma_rn(__dmul_rn(r, r), P, lo));
    if (w >> 54) return 0.0;   // u = 1 (x is 0 only to rounding, of either sign)
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(d2f_chop(x)));
    const double y = f2d_flush(y0), h = f2d_flush(0.5f * y0);
    const double g = __dmul_rn(x, y);
    const double g1 = __fma_rn(g, __fma_rn(-g, h, 0.5), g);
    return __fma_rn(__fma_rn(-g1, g1, x), h, g1);
}

// cos and sin of 2 pi (v + 1/2) 2^-53
__device__ __forceinline__ void noise_turn(const NoiseTable* t, unsigned long long v, double& cs, double& sn) {
    const long long w = (long long)(2ull * v + 1ull);   // 54 bits of a turn
    const long long k = (w + (1ll << 44)) >> 45;        // nearest 512th
    const long long d = w - (k << 45);                  // in [-2^44, 2^44)
    const double2 C = __ldg(reinterpret_cast<const double2*>(t->cs[k & (NOISE_TURN - 1)]));
    // (double)d from the mantissa of 1.5 2^52
    const double dd = __dadd_rn(__longlong_as_double(0x4338000000000000ll + d), -6755399441055744.0);
    const double a = __dmul_rn(dd, 0x1.921fb54442d18p-52);   // 2 pi 2^-54 d, |a| < 2^-7.3
    const double a2 = __dmul_rn(a, a);
    const double sa = __fma_rn(__dmul_rn(a, a2), __fma_rn(a2, 1.0 / 120.0, -1.0 / 6.0), a);
    const float a2f = d2f_chop(a2);
    const float tail = a2f * fmaf(a2f, -1.0f / 720.0f, 1.0f / 24.0f);
    const double cm1 = __dmul_rn(a2, __dadd_rn(f2d_flush(tail), -0.5));   // cos a - 1
    cs = __dadd_rn(C.x, __fma_rn(C.x, cm1, -__dmul_rn(C.y, sa)));
    sn = __dadd_rn(C.y, __fma_rn(C.y, cm1, __dmul_rn(C.x, sa)));
}

// normals 2 b and 2 b + 1 of `atom` at counter `step` for every b < BLOCKS
template <int BLOCKS>
__device__ __forceinline__ void normals(const NoiseTable* t, unsigned long long seed, unsigned long long step,
                                        uint32_t atom, double* out) {
#pragma unroll
    for (uint32_t blk = 0; blk < (uint32_t)BLOCKS; blk++) {
        uint32_t c[4] = {atom, (uint32_t)step, (uint32_t)(step >> 32), blk};
        philox10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
        const double r = noise_radius(t, bits53(c[0], c[1]));
        double cs, sn;
        noise_turn(t, bits53(c[2], c[3]), cs, sn);
        out[2 * blk] = __dmul_rn(r, cs);
        out[2 * blk + 1] = __dmul_rn(r, sn);
    }
}
#endif

}  // namespace parm
