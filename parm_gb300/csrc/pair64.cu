// FP64 pair forces, energies, virials and stresses — the drop-in path whose
// results match the reference CPU code bit for bit.
//
// Reference (wackywendell/parm src/interaction.hpp):
//   NListed<A,P>::set_forces               2165-2175  f_first += F, f_last -= F
//   NListed<A,P>::energy / pressure / stress 2152-2163, 2247-2291
//   LennardJonesCut + LennardJonesCutPair   238-281, 967-987
//   RepulsionPair                           1528-1590
//   LJRepulsive + LJRepulsePair             119-152, 875-891
//   LJAttractCut + LJAttractCutPair         154-236, 1020-1050
//   LoisOhernPair, LoisOhernPairMinCLs      1679-1751
//   LoisLinPair, LoisLinPairMin             1764-1836
//   EisMclachlanPair                        1415-1452
//   RepulsionDragPair                       1598-1640
//   LJAttractRepulseSigsPair                1149-1239
//   indexed epsilons: LennardJonesCutPair / LJAttractCutPair on IEps*Atoms
//   977-982, 1028-1037; LJAttractRepulsePair 1251-1298; LJishPair 1095-1141;
//   LJAttractFixedRepulsePair 1343-1399
//
// Summation order: the reference visits pairs (i, j<i) in ascending (i, j) and
// scatters +F to i and -F to j.  For atom k this is: neighbours j<k in
// ascending j (adding F(k,j)), then neighbours i>k in ascending i
// (subtracting F(i,k)).  Because the minimum image is an exact odd function
// and every pair law scales the displacement by a function of |r|^2,
// -F(i,k) == F(k,i) bit for bit, so gathering F(k, j) over the rank-sorted
// full list reproduces the reference sums exactly.  Pairs beyond the cut-off
// (the reference adds Vec::Zero()) are skipped after an FP32 screen.
//
// Compiled with -fmad=false.
#include "fpbits.cuh"
#include "parm_check.cuh"

namespace parm {

__device__ __forceinline__ bool mobile64(double m) { return !(m <= 0.0 || isinf(m)); }

struct PairC {
    double eps, sig, third, m6;   // the Lois kinds: third = C (or f), m6 = l; LJish: m6 = n
    double cut;                   // the Lois kinds: sigcut; LJAttractRepulse, LJAttractFixedRepulse,
                                  // LJish: the cut energy
    double rep;                   // LJAttractFixedRepulse, LJish: the repulsive epsilon;
                                  // LJAttractRepulseSigs: the attractive one (eps_r in eps,
                                  // sig_a in m6)
    double e12, cut2;             // LJ kinds: 12 eps and cut^2 (set_derived)
    bool safe;                    // 12 eps is 0 or far from overflow and underflow
    __device__ __forceinline__ void set_derived() {
        e12 = 12 * eps;
        cut2 = third * third;
        const uint32_t e = ((uint32_t)__double2hiint(e12) >> 20) & 0x7FFu;
        safe = e12 == 0.0 || (e - 723u < 600u);   // 2^-300 .. 2^300
    }
};

// x > y for y >= 0 and x a sum of squares or a quotient of such (+0, positive,
// +inf or NaN): an integer comparison of the bit patterns, off the FP64 pipe
// (a NaN is not greater)
__device__ __forceinline__ bool above(double x, double y) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return b > (unsigned long long)__double_as_longlong(y) && b <= 0x7FF0000000000000ull;
}

// 12 eps / rsix * (1 / rsix - 1) (LennardJonesCut::forces and its kin, fmagTimesR)
__device__ __forceinline__ double lj_fmag(const PairC& p, double rsix) {
    const double y = 1 / rsix;
    const uint32_t e = ((uint32_t)__double2hiint(rsix) >> 20) & 0x7FFu;
    const double q = (p.safe && e - 723u < 600u) ? quotient_by_reciprocal(p.e12, rsix, y) : p.e12 / rsix;
    return q * (y - 1);
}

// Pair constants of the indexed kinds, A the pair's first atom (the later one
// in the neighbour list: its row of the table is used, IEps*Atom::get_epsilon).
// Atom records: (repeps, sigma, sigcut, p3) with p3 = 1 - 1/sigcut^6
// (LennardJonesCut), LJAttract::energy(sigcut), 1 - sigcut^-6 (the attractive-
// repulsive pairs) or the exponent n (LJish).
template <int KIND>
__device__ __forceinline__ PairC combine_idx(const DevCtx& c, const AtomPrm& A, const AtomPrm& B, uint32_t ta,
                                             uint32_t tb, uint32_t uni) {
    PairC p;
    const uint32_t n = c.ptab_n;
    const double te = c.ptab[(size_t)ta * n + tb];
    p.sig = (uni & IDX_SIG) ? c.ptab[(size_t)n * n + (size_t)ta * n + tb] : (A.p1 + B.p1) / 2.0;
    const bool b_larger = B.p2 > A.p2;
    p.third = b_larger ? B.p2 : A.p2;            // max(a1.sigcut, a2.sigcut)
    const double pc3 = b_larger ? B.p3 : A.p3;   // its per-atom cut term
    p.rep = sqrt(A.p0 * B.p0);
    p.cut = 0.0;
    p.m6 = pc3;
    p.eps = te;
    if constexpr (KIND == KIND_REPULSION_IDX) {
        // RepulsionPair(IEpsISigExpAtom...) (interaction.hpp:1538-1543): the exponent averaged
        p.third = (A.p2 + B.p2) / 2.0;
        p.m6 = 0.0;
    } else if constexpr (KIND == KIND_LJATTRACTREPULSE) {
        if (te <= 0) {
            p.third = 1;
            p.eps = fabs(te);
        } else {
            p.cut = te * (pc3 * pc3);
        }
    } else if constexpr (KIND == KIND_LJFIXEDREPULSE) {
        p.eps = fabs(te);
        if (!(te > 0) || p.eps == 0) {
            p.third = 1;
            p.eps = 0;
        } else {
            p.cut = p.eps * (pc3 * pc3);
        }
    } else if constexpr (KIND == KIND_LJISH) {
        p.m6 = (A.p3 + B.p3) / 2;
        if (te <= 0) {
            p.third = 1;
            p.eps = 0;
        } else {
            const double mid = (1 - pow(p.third, -p.m6));
            p.cut = te * (mid * mid);
        }
    }
    return p;
}

// LJAttractRepulseSigsPair::attract_energy / repulse_energy (interaction.hpp:1192-1202)
__device__ __forceinline__ double sigs_attract(const PairC& p, double r) {
    double r_over_sig = (r - p.sig + p.m6) / p.m6;
    double mid = (1 - pow(r_over_sig, -6.0));
    return p.rep * (mid * mid) - p.rep;
}
__device__ __forceinline__ double sigs_repulse(const PairC& p, double r) {
    double r_over_sig = r / p.sig;
    double mid = (1 - pow(r_over_sig, -6.0));
    return p.eps * (mid * mid) - p.rep;
}

template <int KIND>
__device__ __forceinline__ PairC combine(const AtomPrm& A, const AtomPrm& B, uint32_t uni) {
    PairC p;
    // eps = sqrt(e1*e2) (sqrt(e*e) == e exactly, so uniform epsilon skips it)
    p.eps = (uni & UNI_EPS) ? A.p0 : sqrt(A.p0 * B.p0);
    p.sig = (uni & UNI_SIG) ? A.p1 : (A.p1 + B.p1) / 2;
    if constexpr (cut_kind<KIND>()) {
        // cut = max(a1.sigcut, a2.sigcut); its cut-energy term travels with it
        bool b_larger = B.p2 > A.p2;
        p.third = b_larger ? B.p2 : A.p2;
        p.m6 = b_larger ? B.p3 : A.p3;
    } else if constexpr (KIND == KIND_REPULSION) {
        p.third = (uni & UNI_THIRD) ? A.p2 : (A.p2 + B.p2) / 2.0;
        p.m6 = 0.0;
    } else if constexpr (KIND == KIND_REPULSIONDRAG) {
        // RepulsionDragPair(a1, a2) (interaction.hpp:1613-1621): exponent and gamma averaged
        p.third = (uni & UNI_THIRD) ? A.p2 : (A.p2 + B.p2) / 2.0;
        p.m6 = (uni & UNI_FOURTH) ? A.p3 : (A.p3 + B.p3) / 2;
    } else if constexpr (lois_kind<KIND>()) {
        // LoisOhernPair (interaction.hpp:1693-1703) / LoisLinPair (1782-1800): averages;
        // LoisOhernPairMinCLs (1746-1751) / LoisLinPairMin (1831-1836): the smaller values
        if (uni & COMB_MIN) {
            p.third = A.p2 < B.p2 ? A.p2 : B.p2;
            p.m6 = A.p3 < B.p3 ? A.p3 : B.p3;
        } else {
            p.third = (uni & UNI_THIRD) ? A.p2 : (A.p2 + B.p2) / 2.0;
            p.m6 = (uni & UNI_FOURTH) ? A.p3 : (A.p3 + B.p3) / 2.0;
        }
        // sigcut: sig * (1 + C + l) (LoisOhern), sig + l (LoisLin)
        p.cut = (KIND == KIND_LOISOHERN) ? p.sig * (1 + p.third + p.m6) : p.sig + p.m6;
        return p;
    } else if constexpr (KIND == KIND_LJATTREPSIGS) {
        // LJAttractRepulseSigsPair(a1, a2) (interaction.hpp:1171-1190), atoms (eps_r, eps_a,
        // sig_r, sig_a, sigcut): eps = eps_r, rep = eps_a, sig = sig_r, m6 = sig_a, third =
        // sigcut (max), cut = the cut energy
        p.eps = sqrt(A.p0 * B.p0);
        p.rep = sqrt(A.p1 * B.p1);
        p.sig = (A.p2 + B.p2) / 2.0;
        p.m6 = (A.p3 + B.p3) / 2.0;
        p.third = B.p4 > A.p4 ? B.p4 : A.p4;
        const double cu = p.sig + p.m6 * (p.third - 1);
        p.cut = (p.third >= 1) ? sigs_attract(p, cu) : sigs_repulse(p, cu);
        return p;
    } else if constexpr (KIND == KIND_EISMCLACHLAN) {
        // EisMclachlanPair(a1, a2) (interaction.hpp:1425-1438), atoms (dist, sigmai) =
        // (p0, p1): E = c0/R + c1 + c2 R with c0, c1, c2 in eps, sig, third; cut-off d1 + d2
        p.eps = -M_PI * (A.p1 * B.p0 - B.p1 * A.p0) * (A.p0 * A.p0 - B.p0 * B.p0);
        p.sig = -2 * M_PI * (A.p1 * B.p0 * B.p0 + B.p1 * A.p0 * A.p0);
        p.third = M_PI * (A.p1 * B.p0 + B.p1 * A.p0);
        p.m6 = 0.0;
        p.cut = A.p0 + B.p0;
        return p;
    } else {
        p.third = 0.0;
        p.m6 = 0.0;
    }
    p.cut = 0.0;
    return p;
}

// b^(n - 1) of the soft repulsions: pow(b, 1) == b exactly; the Hertzian
// exponent 5/2 rounded once (three_halves), in a fraction of the FP64 operations of
// the device's pow
__device__ __forceinline__ double power_m1(double b, double n) {
    if (n == 2.0) return b;
    if (n == 2.5) return three_halves(b);
    return pow(b, n - 1);
}

// pair force scale s (F = r * s); returns false beyond the cut-off
template <int KIND>
__device__ __forceinline__ bool force_scale(const PairC& p, double dsq, uint32_t uni, double& s) {
    if constexpr (KIND == KIND_LJATTREPSIGS) {
        // LJAttractRepulseSigsPair::forces (interaction.hpp:1218-1238)
        double cu = p.sig + p.m6 * (p.third - 1);
        if (p.third > 0 && dsq > cu * cu) return false;
        if (dsq > p.sig * p.sig) {
            double dist = sqrt(dsq);
            double rminus = dist - p.sig + p.m6;
            double r_over_sig = rminus / p.m6;
            double rsix = pow(r_over_sig, -6.0);
            double fmag_over_r = 12 * rsix * (rsix - 1) / (dist * rminus);
            s = p.rep * fmag_over_r;
        } else {
            double r_over_sigsq = dsq / (p.sig * p.sig);
            double rsix = pow(r_over_sigsq, -3.0);
            double fmagTimesR = 12 * rsix * (rsix - 1);
            s = p.eps * fmagTimesR / dsq;
        }
        return true;
    } else if constexpr (KIND == KIND_LJATTRACTREPULSE) {
        // LJAttractRepulsePair::forces (interaction.hpp:1287-1297)
        if (p.eps == 0) return false;
        double rsq = dsq / (p.sig * p.sig);
        if (rsq > (p.third * p.third)) return false;
        double rsix = pow(rsq, -3.0);
        double fmagTimesR = 12 * p.eps * rsix * (rsix - 1);
        s = fmagTimesR / dsq;
        return true;
    } else if constexpr (KIND == KIND_LJFIXEDREPULSE || KIND == KIND_LJISH) {
        // LJAttractFixedRepulsePair::forces (1390-1398), LJishPair::forces (1130-1140)
        double rsq = dsq / (p.sig * p.sig);
        if (rsq > (p.third * p.third)) return false;
        double fmagTimesR;
        if constexpr (KIND == KIND_LJFIXEDREPULSE) {
            double rsix = pow(rsq, -3.0);
            fmagTimesR = 12 * rsix * (rsix - 1);
        } else {
            double n = p.m6;
            double rmid = pow(rsq, -n / 2);
            fmagTimesR = 2 * n * rmid * (rmid - 1);
        }
        s = (rsq < 1) ? p.rep * fmagTimesR / dsq : p.eps * fmagTimesR / dsq;
        return true;
    } else if constexpr (KIND == KIND_LJCUT || KIND == KIND_LJCUT_IDX) {
        double rsq = (uni & UNI_SIG_ONE) ? dsq : dsq / (p.sig * p.sig);
        if (above(rsq, p.cut2)) return false;
        double rsix = rsq * rsq * rsq;
        s = lj_fmag(p, rsix) / dsq;
        return true;
    } else if constexpr (KIND == KIND_REPULSION || KIND == KIND_REPULSION_IDX) {
        if (above(dsq, p.sig * p.sig)) return false;
        double R = sqrt(dsq);
        double b = 1.0 - (R / p.sig);
        double pw = power_m1(b, p.third);
        s = p.eps * pw / p.sig / R;
        return true;
    } else if constexpr (KIND == KIND_LJATTRACT || KIND == KIND_LJATTRACT_IDX) {
        // LJAttractCut::forces (interaction.hpp:219-229)
        if (p.eps == 0) return false;
        double rsq = (uni & UNI_SIG_ONE) ? dsq : dsq / (p.sig * p.sig);
        if (rsq < 1 || above(rsq, p.cut2)) return false;
        double rsix = rsq * rsq * rsq;
        s = lj_fmag(p, rsix) / dsq;
        return true;
    } else if constexpr (KIND == KIND_LOISOHERN) {
        // LoisOhernPair::forces (interaction.hpp:1729-1743): harmonic to (1 + C) sigma,
        // then a linear return to zero at sigcut
        const double C = p.third, l = p.m6;
        if (dsq >= p.cut * p.cut) return false;
        double R = sqrt(dsq);
        double rsig = R / p.sig;
        if (rsig <= 1 + C) {
            double dR = rsig - 1;
            s = -p.eps * dR / R;
        } else {
            double dR2 = rsig - (C + l + 1);
            s = C * p.eps / l * dR2 / R;
        }
        return true;
    } else if constexpr (KIND == KIND_EISMCLACHLAN) {
        // EisMclachlanPair::forces (interaction.hpp:1445-1451)
        if (dsq > (p.cut * p.cut)) return false;
        double R = sqrt(dsq);
        s = (p.eps / dsq - p.third) / R;
        return true;
    } else if constexpr (KIND == KIND_LOISLIN) {
        // LoisLinPair::forces (interaction.hpp:1817-1828); -rij * (f / R) == rij * -(f / R)
        if (dsq >= p.cut * p.cut) return false;
        double R = sqrt(dsq);
        if (R <= p.sig) {
            double dR = 1.0 - (R / p.sig);
            s = p.eps * dR / p.sig / R;
        } else {
            s = -(p.third / R);
        }
        return true;
    } else {
        double rsq = (uni & UNI_SIG_ONE) ? dsq : dsq / (p.sig * p.sig);
        if (above(rsq, 1.0)) return false;
        double rsix = rsq * rsq * rsq;
        s = lj_fmag(p, rsix) / dsq;
        return true;
    }
}

template <int KIND>
__device__ __forceinline__ double pair_energy(const PairC& p, double dsq, uint32_t uni) {
    if constexpr (KIND == KIND_LJATTREPSIGS) {
        // LJAttractRepulseSigsPair::energy (interaction.hpp:1204-1216)
        double dist = sqrt(dsq);
        double cu = p.sig + p.m6 * (p.third - 1);
        if (p.third > 0 && dist > cu) return 0.0;
        if (dist <= p.sig) return sigs_repulse(p, dist) - p.cut;
        return sigs_attract(p, dist) - p.cut;
    } else if constexpr (KIND == KIND_LJATTRACTREPULSE || KIND == KIND_LJFIXEDREPULSE || KIND == KIND_LJISH) {
        // LJAttractRepulsePair::energy (1269-1286), LJAttractFixedRepulsePair::energy (1366-1389),
        // LJishPair::energy (1115-1129)
        double rsq = dsq / (p.sig * p.sig);
        if (rsq > p.third * p.third) return 0.0;
        double mid = (KIND == KIND_LJISH) ? (1 - pow(rsq, -p.m6 / 2)) : (1 - pow(rsq, -3.0));
        if constexpr (KIND == KIND_LJATTRACTREPULSE) return p.eps * (mid * mid) - p.cut;
        if (rsq > 1) return p.eps * (mid * mid) - p.cut;
        return p.rep * (mid * mid) - p.cut;
    } else if constexpr (KIND == KIND_LJCUT || KIND == KIND_LJCUT_IDX) {
        double rsq = (uni & UNI_SIG_ONE) ? dsq : dsq / (p.sig * p.sig);
        if (rsq > (p.third * p.third)) return 0.0;
        double rsix = rsq * rsq * rsq;
        double mid = (1 - 1 / rsix);
        double cut_energy = p.eps * (p.m6 * p.m6 - 1);
        return p.eps * (mid * mid - 1) - cut_energy;
    } else if constexpr (KIND == KIND_REPULSION || KIND == KIND_REPULSIONDRAG || KIND == KIND_REPULSION_IDX) {
        // RepulsionPair::energy (1544-1550), RepulsionDragPair::energy (1622-1628)
        if (dsq > p.sig * p.sig) return 0.0;
        double R = sqrt(dsq);
        double b = 1.0 - (R / p.sig);
        double pw = (p.third == 2.0) ? b * b : pow(b, p.third);   // pow(b, 2) == b*b exactly
        return p.eps * pw / p.third;
    } else if constexpr (KIND == KIND_LJATTRACT || KIND == KIND_LJATTRACT_IDX) {
        // LJAttractCut::energy (interaction.hpp:211-216) with LJAttract::energy (162-169)
        if (p.eps == 0) return 0.0;
        if (dsq > (p.third * p.third * p.sig * p.sig)) return 0.0;
        double rsq = dsq / (p.sig * p.sig);
        double e;
        if (rsq < 1) {
            e = -p.eps;
        } else {
            double rsix = rsq * rsq * rsq;
            double mid = (1 - 1 / rsix);
            e = p.eps * (mid * mid - 1);
        }
        return e - p.m6 * p.eps;
    } else if constexpr (KIND == KIND_LOISOHERN) {
        // LoisOhernPair::energy (interaction.hpp:1713-1727)
        const double C = p.third, l = p.m6;
        if (dsq >= p.cut * p.cut) return 0.0;
        double R = sqrt(dsq) / p.sig;
        if (R <= 1 + C) {
            double dR = R - 1;
            return -p.eps * p.sig / 2 * (C * (C + l) - dR * dR);
        }
        double dR2 = C + l + 1 - R;
        return -C * p.eps * p.sig / 2 / l * dR2 * dR2;
    } else if constexpr (KIND == KIND_EISMCLACHLAN) {
        // EisMclachlanPair::energy (interaction.hpp:1439-1444)
        double R = sqrt(dsq);
        if (R > p.cut) return 0.0;
        return p.eps / R + p.sig + p.third * R;
    } else if constexpr (KIND == KIND_LOISLIN) {
        // LoisLinPair::energy (interaction.hpp:1802-1815)
        const double f = p.third, l = p.m6;
        if (dsq >= p.cut * p.cut) return 0.0;
        double R = sqrt(dsq);
        if (R <= p.sig) {
            double dR = 1.0 - (R / p.sig);
            return p.eps / 2 * dR * dR - f * l;
        }
        return -f * (p.sig + l - R);
    } else {
        double rsq = (uni & UNI_SIG_ONE) ? dsq : dsq / (p.sig * p.sig);
        if (rsq > 1) return 0.0;
        double rsix = rsq * rsq * rsq;
        double mid = (1 - 1 / rsix);
        return p.eps * (mid * mid);
    }
}

// RepulsionDragPair::forces (interaction.hpp:1629-1639): the soft repulsion
// minus gamma times the relative velocity's component along r; false beyond
// the cut-off.  F(i, j) == -F(j, i) bit for bit (r and v_i - v_j both flip).
template <int ND>
__device__ __forceinline__ bool drag_force(const PairC& p, const double* r, double dsq, const double* vi,
                                           const double* vj, double* fo) {
    if (dsq > p.sig * p.sig) return false;
    double R = sqrt(dsq);
    double vij[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < ND; d++) vij[d] = vi[d] - vj[d];
    double vdot = vij[0] * r[0] + vij[1] * r[1];
    if constexpr (ND == 3) vdot = vdot + vij[2] * r[2];
    double b = 1.0 - (R / p.sig);
    double pw = power_m1(b, p.third);
    double sr = p.eps * pw / p.sig / R;
#pragma unroll
    for (int d = 0; d < ND; d++) {
        double vperp = r[d] * vdot / dsq;
        fo[d] = r[d] * sr - vperp * p.m6;
    }
    return true;
}

// FP32 screen: true when the pair is certainly beyond the cut-off
// (Q = (sqrt(eps), sigma, third, fourth) in FP32)
template <int KIND>
__device__ __forceinline__ bool beyond32(float d2, const float4& Qi, const float4& Qj, uint32_t uni) {
    if constexpr (idx_kind<KIND>() || KIND == KIND_LJATTREPSIGS) return false;   // every pair takes the exact test
    float sg = (uni & UNI_SIG) ? Qi.y : 0.5f * (Qi.y + Qj.y);
    float rc;
    if constexpr (cut_kind<KIND>()) {
        rc = sg * fmaxf(Qi.z, Qj.z);
    } else if constexpr (lois_kind<KIND>()) {
        const bool mn = uni & COMB_MIN;
        const float th = mn ? fminf(Qi.z, Qj.z) : 0.5f * (Qi.z + Qj.z);
        const float l = mn ? fminf(Qi.w, Qj.w) : 0.5f * (Qi.w + Qj.w);
        rc = (KIND == KIND_LOISOHERN) ? sg * (1.0f + th + l) : sg + l;
    } else if constexpr (KIND == KIND_EISMCLACHLAN) {
        rc = Qi.x + Qj.x;   // dist_i + dist_j
    } else {
        rc = sg;
    }
    return d2 > rc * rc * 1.0002f;
}

template <int ND>
__device__ __forceinline__ void load3(const void* p, uint32_t i, double* o) {
    using V = typename DVec<ND>::T;
    V t = static_cast<const V*>(p)[i];
    const double* q = reinterpret_cast<const double*>(&t);
#pragma unroll
    for (int d = 0; d < ND; d++) o[d] = q[d];
}

template <int ND>
__device__ __forceinline__ void store3(void* p, uint32_t i, const double* o) {
    using V = typename DVec<ND>::T;
    V t;
    double* q = reinterpret_cast<double*>(&t);
#pragma unroll
    for (int d = 0; d < (int)(sizeof(V) / 8); d++) q[d] = d < ND ? o[d] : 0.0;
    static_cast<V*>(p)[i] = t;
}

// FP32 squared distance of the minimum image, 0 when the image is in doubt:
// disp32 picks it from the coarse parts, which can be off by 1/8, so near half
// a box length it may take the farther one, and beyond 2^20 the coarse parts
// and their difference are no longer exact.  `wrap` tells whether the FP64
// displacement needs the remainder.  It does not when every component is well
// below half a box length without a shift: |x_i - x_j| < L/2 is its own
// remainder (the FP32 components are within an ulp or so of the FP64 ones).
template <int ND>
__device__ __forceinline__ float image32(const SysConst& S, const float4& Ai, const float4& Bi, const float4& Aj,
                                         const float4& Bj, bool& wrap) {
    const float Xi[3] = {Ai.x, Ai.y, Ai.z}, Xj[3] = {Aj.x, Aj.y, Aj.z};
    const float Fi[3] = {Bi.x, Bi.y, Bi.z}, Fj[3] = {Bj.x, Bj.y, Bj.z};
    float d2 = 0.f;
    bool doubt = false;
    wrap = false;
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const float r = disp32(Xi[d], Xj[d], Fi[d], Fj[d], S.Lhi[d], S.Llo[d], S.invLf[d]);
        d2 += r * r;
        doubt = doubt || fabsf(r) > 0.499f * S.Lhi[d] - 0.13f || !(fabsf(Xi[d]) < 1048576.0f) ||
                !(fabsf(Xj[d]) < 1048576.0f);
        wrap = wrap || !(fabsf((Xi[d] - Xj[d]) + (Fi[d] - Fj[d])) < 0.49f * S.Lhi[d]);
    }
    wrap = wrap || doubt;
    return doubt ? 0.f : d2;
}

// ---------------------------------------------------------------------------
// Forces.  What bounds them: the FP64 pipe (2 lanes per clock and SM), about
// 40 FP64 operations per interacting LJ pair; so the FP64 part runs on full
// warps of pairs that pass an FP32 screen, each pair once where memory allows.
//
// Pair forces kept (launch_force64 with c.pairf set): k_pair64 evaluates every
// listed pair once, for its first atom (the one of higher rank: its list
// entries below half_n), and writes the force to the pair's slot; k_sum64 adds
// each atom's slots in list order, its own pairs and then, negated, those of
// the atoms ranked after it: the reference's order and its f_last -= F.
//
// Without (handles whose slots would take too much memory): k_force64
// evaluates every pair for both of its atoms, so it needs no slots.
//
// A CTA takes F64_ATOMS consecutive atoms in rounds of F64_CHUNK list entries:
// a warp per atom screens the entries, 32 at a time, and appends the survivors
// to the atom's segment in list order; the CTA's survivors are then numbered
// consecutively and evaluated one per thread.  A pair that turns out not to
// interact adds +0, which changes no sum that starts at +0.
// Measured, LJ, ~72 listed pairs per atom (one GB300): a thread per atom that
// walked its list 379 us at 1000 atoms, 385 us at 29,667, 8.03 ms at 1,048,576
// (a third of its lanes idle in the FP64 part, a serial chain over the list);
// k_force64 23.4 us, 161 us, 4.39 ms; k_pair64 + k_sum64 114 us at 29,667 and
// 3.10 ms at 1,048,576 (k_pair64: FP64 pipe 85 % busy).
// ---------------------------------------------------------------------------
constexpr int F64_THREADS = 128;
constexpr uint32_t F64_ATOMS = 8;    // x 3 components: the lanes of k_force64's summing warp
constexpr uint32_t F64_CHUNK = 96;   // list entries per atom and round (whole LJ lists in one round)
constexpr uint32_t F64_SEG = F64_CHUNK + 1;   // odd: the summing lanes read different banks

// FP32 screen of entry (i, j): false when the pair is certainly beyond the cut-off
template <int ND, int KIND>
__device__ __forceinline__ bool screen64(const DevCtx& c, const SysConst& S, const float4& Ai, const float4& Bi,
                                         const float4& Qi, uint32_t j, bool& wrap) {
    float4 Aj, Bj;
    ld_pos_coherent(c.pos, j, Aj, Bj);
    float4 Qj = Qi;
    if ((c.uniform & UNI_ALL) != UNI_ALL) Qj = c.prm32[j];
    // (the screen is per-axis periodic: not for a sheared box)
    const float d2 = image32<ND>(S, Ai, Bi, Aj, Bj, wrap);
    return S.lees || !beyond32<KIND>(d2, Qi, Qj, c.uniform);
}

// pair constants of (i, j); `first` tells that i is the pair's first atom
template <int KIND>
__device__ __forceinline__ PairC pair_constants(const DevCtx& c, uint32_t i, uint32_t j, bool first) {
    const uint32_t uni = c.uniform;
    const AtomPrm Pi = c.prm[i];
    PairC pc;
    if constexpr (idx_kind<KIND>()) {
        const uint32_t ti = __float_as_uint(c.prm32[i].x), tj = __float_as_uint(c.prm32[j].x);
        pc = first ? combine_idx<KIND>(c, Pi, c.prm[j], ti, tj, uni) : combine_idx<KIND>(c, c.prm[j], Pi, tj, ti, uni);
    } else {
        pc = combine<KIND>(Pi, (uni & UNI_ALL) == UNI_ALL ? Pi : c.prm[j], uni);
    }
    pc.set_derived();
    return pc;
}

// FP64 force of j on i (0 beyond the cut-off); `wrap`: the minimum image needs the remainder
template <int ND, int KIND>
__device__ __forceinline__ void force_of_pair(const DevCtx& c, const SysConst& S, uint32_t i, uint32_t j,
                                              const double* xi, bool wrap, const PairC& pc, double* fo) {
    double xj[3] = {0, 0, 0}, r[3] = {0, 0, 0};
    load3<ND>(c.x, j, xj);
    if (S.lees) {
        lees_diff<ND>(S, xi, xj, r);
    } else {
#pragma unroll
        for (int d = 0; d < ND; d++) r[d] = xi[d] - xj[d];
        if (wrap) {
#pragma unroll
            for (int d = 0; d < ND; d++) r[d] = remainder_exact(r[d], S.L[d], S.invL[d], S.halfL[d]);
        }
    }
    double dsq = r[0] * r[0] + r[1] * r[1];
    if constexpr (ND == 3) dsq = dsq + r[2] * r[2];
    fo[0] = fo[1] = fo[2] = 0.0;
    if constexpr (KIND == KIND_REPULSIONDRAG) {
        double vi[3] = {0, 0, 0}, vj[3] = {0, 0, 0};
        load3<ND>(c.v, i, vi);
        load3<ND>(c.v, j, vj);
        if (!drag_force<ND>(pc, r, dsq, vi, vj, fo)) fo[0] = fo[1] = fo[2] = 0.0;
    } else {
        double sc;
        if (force_scale<KIND>(pc, dsq, c.uniform, sc)) {
#pragma unroll
            for (int d = 0; d < ND; d++) fo[d] = r[d] * sc;
        }
    }
}

// f of internal atom i and, with MODE FM_FORCES_A, a = f/m (Collection::
// set_forces(true): zero for m <= 0 or inf)
template <int ND, int MODE>
__device__ __forceinline__ void store_force(const DevCtx& c, uint32_t i, const double* f) {
    store3<ND>(c.f, i, f);
    if constexpr (MODE == FM_FORCES_A) {
        const double m = c.m[i];
        double a[3] = {0, 0, 0};
        if (mobile64(m)) {
#pragma unroll
            for (int d = 0; d < ND; d++) a[d] = f[d] / m;
        }
        store3<ND>(c.a, i, a);
    }
}

// a pair force's slot: one 32-byte (2D: 16-byte) access
template <int ND> struct SlotVec;
template <> struct SlotVec<3> { using T = double4_32a; };
template <> struct SlotVec<2> { using T = double2; };

// The work of k_pair64 (HALF) and k_force64.
template <int ND, int KIND, int MODE, bool HALF>
__device__ __forceinline__ void forces64(const DevCtx& c) {
    __shared__ double pf[HALF ? 1 : ND][HALF ? 1 : F64_ATOMS * F64_SEG];   // pair forces
    __shared__ uint32_t pj[F64_ATOMS * F64_CHUNK];      // surviving neighbours
    __shared__ uint8_t pw[F64_ATOMS * F64_CHUNK];       // 1: the minimum image needs the remainder
    __shared__ uint16_t pk[HALF ? F64_ATOMS * F64_CHUNK : 1];   // their list entries
    __shared__ double xs[F64_ATOMS][4];
    __shared__ uint32_t nn_s[F64_ATOMS], cnt[F64_ATOMS], slot0[F64_ATOMS];
    using V = typename SlotVec<ND>::T;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t i0 = blockIdx.x * F64_ATOMS;
    const bool all_uni = (c.uniform & UNI_ALL) == UNI_ALL;
    release_next();
    // (list lengths and ranks do not change in the drift before)
    bool go = false;
    if (tid < F64_ATOMS) {
        const uint32_t i = i0 + tid;
        go = i < c.n && c.active[c.atom_sys[i]] && c.rank[i] != NOT_MEMBER;
        nn_s[tid] = !go ? 0u : (HALF ? c.half_n[i] : c.nnb[i]);
        slot0[tid] = HALF && go ? c.half_base[i] : 0u;
    }
    wait_previous();
    if (tid < F64_ATOMS) {
        const uint32_t i = i0 + tid;
        double xi[3] = {0, 0, 0};
        if (go) load3<ND>(c.x, i, xi);
#pragma unroll
        for (int d = 0; d < 3; d++) xs[tid][d] = xi[d];
    }
    __syncthreads();
    uint32_t nmax = 0;
#pragma unroll
    for (uint32_t a = 0; a < F64_ATOMS; a++) nmax = max(nmax, nn_s[a]);
    const uint32_t sa = tid % F64_ATOMS, sd = tid / F64_ATOMS;   // summing lane: atom, component
    double fsum = 0.0;
    PairC pc;
    bool have = false;
    for (uint32_t base = 0; base < nmax; base += F64_CHUNK) {
        for (uint32_t a = warp; a < F64_ATOMS; a += F64_THREADS / 32) {
            const uint32_t hi = min(nn_s[a], base + F64_CHUNK);
            uint32_t m = 0;
            if (base < hi) {
                const uint32_t i = i0 + a;
                const SysConst& S = c.sys[c.atom_sys[i]];
                const uint32_t* nb = c.nbr + (size_t)i * c.maxnb;
                float4 Ai, Bi;
                ld_pos_coherent(c.pos, i, Ai, Bi);
                const float4 Qi = c.prm32[i];
                for (uint32_t k0 = base; k0 < hi; k0 += 32u) {
                    const uint32_t k = k0 + lane;
                    bool keep = false, wrap = true;
                    uint32_t j = 0;
                    if (k < hi) {
                        j = __ldg(nb + k);
                        keep = screen64<ND, KIND>(c, S, Ai, Bi, Qi, j, wrap);
                        if (HALF && !keep) static_cast<V*>(c.pairf)[slot0[a] + k] = V{};
                    }
                    const uint32_t mask = __ballot_sync(0xFFFFFFFFu, keep);
                    if (keep) {
                        const uint32_t q = a * F64_CHUNK + m + __popc(mask & ((1u << lane) - 1u));
                        pj[q] = j;
                        pw[q] = wrap ? 1 : 0;
                        if (HALF) pk[q] = (uint16_t)k;
                    }
                    m += __popc(mask);
                }
            }
            if (lane == 0) cnt[a] = m;
        }
        __syncthreads();
        uint32_t total = 0;
#pragma unroll
        for (uint32_t a = 0; a < F64_ATOMS; a++) total += cnt[a];
        for (uint32_t t = tid; t < total; t += F64_THREADS) {
            uint32_t a = 0, m = t;
            while (m >= cnt[a]) m -= cnt[a++];
            const uint32_t q = a * F64_CHUNK + m, i = i0 + a, j = pj[q];
            if (!all_uni || !have) {
                pc = pair_constants<KIND>(c, i, j, HALF || c.rank[i] > c.rank[j]);
                have = true;
            }
            double fo[3];
            force_of_pair<ND, KIND>(c, c.sys[c.atom_sys[i]], i, j, xs[a], pw[q] != 0, pc, fo);
            if constexpr (HALF) {
                V v;
                double* vp = reinterpret_cast<double*>(&v);
#pragma unroll
                for (int d = 0; d < (int)(sizeof(V) / 8); d++) vp[d] = d < ND ? fo[d] : 0.0;
                static_cast<V*>(c.pairf)[slot0[a] + pk[q]] = v;
            } else {
#pragma unroll
                for (int d = 0; d < ND; d++) pf[HALF ? 0 : d][a * F64_SEG + m] = fo[d];
            }
        }
        __syncthreads();
        if constexpr (!HALF) {
            if (sd < ND) {
                const double* p = &pf[sd][sa * F64_SEG];
                const uint32_t m = cnt[sa];
#pragma unroll 4
                for (uint32_t k = 0; k < m; k++) fsum = fsum + p[k];
            }
            __syncthreads();
        }
    }
    if constexpr (!HALF) {
        // the components of an atom meet in its segment
        if (sd < ND) pf[sd][sa * F64_SEG] = fsum;
        __syncthreads();
        const uint32_t i = i0 + tid;
        if (tid >= F64_ATOMS || i >= c.n || !c.active[c.atom_sys[i]]) return;
        double f[3] = {0, 0, 0};
#pragma unroll
        for (int d = 0; d < ND; d++) f[d] = pf[d][tid * F64_SEG];
        store_force<ND, MODE>(c, i, f);
    }
}

template <int ND, int KIND, int MODE>
__global__ void __launch_bounds__(F64_THREADS) k_force64(DevCtx c) {
    forces64<ND, KIND, MODE, false>(c);
}

// k_force64 for short lists (a warp per atom would leave most lanes idle in
// the screen, and eight atoms too few survivors for a warp): F64S_ATOMS atoms
// a CTA, their entries numbered consecutively and screened one per thread, the
// survivors evaluated one per thread in any order, each force stored at its
// entry's place, and every entry added in order, zeros included (nothing is
// added where no pair of the CTA survives).
// FP64-bound from there (a soft-sphere pair takes ~55 FP64 operations): k_force64 /
// this 54.8 / 42.9 us on 65,536 harmonic disks, 34.5 / 30.1 us on 20,000 spheres.
constexpr int F64S_THREADS = 128;
constexpr uint32_t F64S_ATOMS = 16, F64S_CHUNK = 32;   // entries per atom and round
constexpr uint32_t F64S_CAP = F64S_ATOMS * F64S_CHUNK;
template <int ND, int KIND, int MODE>
__global__ void __launch_bounds__(F64S_THREADS) k_force64s(DevCtx c) {
    __shared__ double pf[ND][F64S_CAP];                 // pair forces by entry
    __shared__ uint32_t pj[F64S_CAP];                   // survivors: neighbour,
    __shared__ uint16_t pe[F64S_CAP];                   // entry,
    __shared__ uint8_t pa[F64S_CAP];                    // atom | 128 when the image needs the remainder
    __shared__ double xs[F64S_ATOMS][4];
    __shared__ uint32_t off[F64S_ATOMS + 1], nsurv;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    const uint32_t i0 = blockIdx.x * F64S_ATOMS;
    const bool all_uni = (c.uniform & UNI_ALL) == UNI_ALL;
    release_next();
    uint32_t nn = 0u, nmax = 0u;   // of atom i0 + lane, in every warp
    {
        const uint32_t i = i0 + lane;
        const bool go = lane < F64S_ATOMS && i < c.n && c.active[c.atom_sys[i]] && c.rank[i] != NOT_MEMBER;
        if (go) nn = c.nnb[i];
        nmax = __reduce_max_sync(0xFFFFFFFFu, nn);
        wait_previous();
        if (tid < F64S_ATOMS) {
            double xi[3] = {0, 0, 0};
            if (go) load3<ND>(c.x, i, xi);
#pragma unroll
            for (int d = 0; d < 3; d++) xs[lane][d] = xi[d];
        }
    }
    constexpr uint32_t SUMS = F64S_ATOMS * ND;   // (atom, component) pairs, one per thread
    const uint32_t sa = tid % F64S_ATOMS, sd = tid / F64S_ATOMS;
    double fsum = 0.0;
    PairC pc;
    bool have = false;
    for (uint32_t base = 0; base < nmax; base += F64S_CHUNK) {
        if (tid < 32u) {
            const uint32_t m = nn > base ? min(nn - base, F64S_CHUNK) : 0u;
            uint32_t incl = m;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += u;
            }
            if (lane < F64S_ATOMS) off[lane + 1] = incl;
            if (lane == 0) off[0] = nsurv = 0u;
        }
        __syncthreads();
        const uint32_t total = off[F64S_ATOMS];
        for (uint32_t t0 = tid - lane; t0 < total; t0 += F64S_THREADS) {   // uniform in the warp
            const uint32_t t = t0 + lane;
            bool keep = false, wrap = true;
            uint32_t a = 0u, j = 0u;
            if (t < total) {
#pragma unroll
                for (uint32_t h = F64S_ATOMS / 2; h; h >>= 1)
                    if (off[a + h] <= t) a += h;
                const uint32_t i = i0 + a;
                j = __ldg(c.nbr + (size_t)i * c.maxnb + base + (t - off[a]));
                float4 Ai, Bi;
                ld_pos_coherent(c.pos, i, Ai, Bi);
                keep = screen64<ND, KIND>(c, c.sys[c.atom_sys[i]], Ai, Bi, c.prm32[i], j, wrap);
                if (!keep) {
#pragma unroll
                    for (int d = 0; d < ND; d++) pf[d][t] = 0.0;
                }
            }
            const uint32_t mask = __ballot_sync(0xFFFFFFFFu, keep);
            uint32_t q = 0u;
            if (lane == 0 && mask) q = atomicAdd(&nsurv, (uint32_t)__popc(mask));
            q = __shfl_sync(0xFFFFFFFFu, q, 0) + __popc(mask & ((1u << lane) - 1u));
            if (keep) {
                pj[q] = j;
                pe[q] = (uint16_t)t;
                pa[q] = (uint8_t)(a | (wrap ? 128u : 0u));
            }
        }
        __syncthreads();
        const uint32_t ns = nsurv;
        if (ns == 0u) {   // (no pair of the CTA interacts: nothing to add)
            if (base + F64S_CHUNK < nmax) __syncthreads();
            continue;
        }
        for (uint32_t q = tid; q < ns; q += F64S_THREADS) {
            const uint32_t a = pa[q] & 127u, i = i0 + a, j = pj[q];
            if (!all_uni || !have) {
                pc = pair_constants<KIND>(c, i, j, c.rank[i] > c.rank[j]);
                have = true;
            }
            double fo[3];
            force_of_pair<ND, KIND>(c, c.sys[c.atom_sys[i]], i, j, xs[a], (pa[q] & 128u) != 0u, pc, fo);
#pragma unroll
            for (int d = 0; d < ND; d++) pf[d][pe[q]] = fo[d];
        }
        __syncthreads();
        if (tid < SUMS) {
            const uint32_t hi = off[sa + 1];
#pragma unroll 4
            for (uint32_t t = off[sa]; t < hi; t++) fsum = fsum + pf[sd][t];
        }
        __syncthreads();
    }
    __syncthreads();
    // the components of an atom meet in shared memory
    if (tid < SUMS) pf[sd][sa] = fsum;
    __syncthreads();
    const uint32_t i = i0 + tid;
    if (tid >= F64S_ATOMS || i >= c.n || !c.active[c.atom_sys[i]]) return;
    double f[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < ND; d++) f[d] = pf[d][tid];
    store_force<ND, MODE>(c, i, f);
}
// k_force64 for many atoms: a warp per 32 of them, on its own.  Every lane screens
// its atom's list, the survivors are numbered consecutively (in list order by
// atom) and evaluated one per lane, each lane then adds its atom's in order.  No
// barrier and little work besides the screen, which is all there is to do where
// few listed pairs interact; its latencies need some fifteen warps an SM.
// k_force64s / k_force64w, WCA just below contact: 25.5 / 15.5 us at 80,000 atoms
// in 2D, 175 / 67 us at 600,000, 242 / 123 us in 3D (a thread per atom that
// walked its list 16, 66 and 175 us); 48 WCA replicas (427,107 atoms) 270 / 191
// us, 400,000 disks 243 / 199 us; but 100,000 overlapping spheres 102 / 117 us,
// 65,536 disks 42 / 48 us.  Lists of 55 entries, of which a few interact:
// k_force64 / k_force64w 95 / 79 us at 80,000 spheres, 521 / 319 us at 400,000.
constexpr int F64W_WARPS = 4;
constexpr uint32_t F64W_CHUNK = 16, F64W_BATCH = 128;   // list entries per atom and round; pair forces held at once
template <int ND, int KIND, int MODE>
__global__ void __launch_bounds__(32 * F64W_WARPS) k_force64w(DevCtx c) {
    __shared__ double pf_s[F64W_WARPS][ND][F64W_BATCH];
    __shared__ double xs_s[F64W_WARPS][ND][32];
    __shared__ uint32_t pj_s[F64W_WARPS][32u * F64W_CHUNK];   // survivors: neighbour,
    __shared__ uint8_t pa_s[F64W_WARPS][32u * F64W_CHUNK];    // atom | 128 when the image needs the remainder
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t i0 = (blockIdx.x * F64W_WARPS + warp) * 32u, i = i0 + lane;
    release_next();
    // (list lengths, lists and ranks do not change in the drift before)
    const bool all_uni = (c.uniform & UNI_ALL) == UNI_ALL;
    const uint32_t s = i < c.n ? c.atom_sys[i] : 0u;
    const bool live = i < c.n && c.active[s];
    const uint32_t nn = live && c.rank[i] != NOT_MEMBER ? c.nnb[i] : 0u;
    const uint32_t nmax = __reduce_max_sync(0xFFFFFFFFu, nn);
    const SysConst& S = c.sys[s];
    double (*pf)[F64W_BATCH] = pf_s[warp];
    double (*xs)[32] = xs_s[warp];
    uint32_t* pj = pj_s[warp];
    uint8_t* pa = pa_s[warp];
    wait_previous();
    float4 Ai, Bi, Qi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (nn) {
        double xi[3] = {0, 0, 0};
        load3<ND>(c.x, i, xi);
#pragma unroll
        for (int d = 0; d < ND; d++) xs[d][lane] = xi[d];
        ld_pos_coherent(c.pos, i, Ai, Bi);
        Qi = c.prm32[i];
    }
    const uint4* row = reinterpret_cast<const uint4*>(c.nbr + (size_t)i * c.maxnb);   // (maxnb: a multiple of 8)
    double f[3] = {0, 0, 0};
    PairC pc;
    bool have = false;
    for (uint32_t base = 0; base < nmax; base += F64W_CHUNK) {
        uint32_t keep = 0u, wraps = 0u;
        uint4 J[F64W_CHUNK / 4];
#pragma unroll
        for (uint32_t g = 0; g < F64W_CHUNK / 4; g++)
            J[g] = base + 4u * g < nn ? __ldg(row + (base >> 2) + g) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (uint32_t g = 0; g < F64W_CHUNK / 4; g++) {
            if (base + 4u * g >= nmax) break;   // uniform in the warp
            const uint32_t js[4] = {J[g].x, J[g].y, J[g].z, J[g].w};
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                bool wrap;
                if (base + 4u * g + u < nn && screen64<ND, KIND>(c, S, Ai, Bi, Qi, js[u], wrap)) {
                    keep |= 1u << (4u * g + u);
                    wraps |= (wrap ? 1u : 0u) << (4u * g + u);
                }
            }
        }
        uint32_t end = __popc(keep);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, end, o);
            if (lane >= (uint32_t)o) end += u;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, end, 31), first = end - __popc(keep);
        uint32_t q = first;
#pragma unroll
        for (uint32_t g = 0; g < F64W_CHUNK / 4; g++) {
            const uint32_t js[4] = {J[g].x, J[g].y, J[g].z, J[g].w};
#pragma unroll
            for (uint32_t u = 0; u < 4; u++) {
                if ((keep >> (4u * g + u)) & 1u) {
                    pj[q] = js[u];
                    pa[q] = (uint8_t)(lane | (((wraps >> (4u * g + u)) & 1u) << 7));
                    q++;
                }
            }
        }
        __syncwarp();
        for (uint32_t b0 = 0; b0 < total; b0 += F64W_BATCH) {
            const uint32_t b1 = min(total, b0 + F64W_BATCH);
            for (uint32_t t = b0 + lane; t < b1; t += 32u) {
                const uint32_t w = pa[t], a = w & 31u, ia = i0 + a, j = pj[t];
                if (!all_uni || !have) {
                    pc = pair_constants<KIND>(c, ia, j, c.rank[ia] > c.rank[j]);
                    have = true;
                }
                double xi[3] = {0, 0, 0}, fo[3];
#pragma unroll
                for (int d = 0; d < ND; d++) xi[d] = xs[d][a];
                force_of_pair<ND, KIND>(c, c.sys[c.atom_sys[ia]], ia, j, xi, (w & 128u) != 0u, pc, fo);
#pragma unroll
                for (int d = 0; d < ND; d++) pf[d][t - b0] = fo[d];
            }
            __syncwarp();
            const uint32_t hi = min(end, b1);
            for (uint32_t t = max(first, b0); t < hi; t++) {
#pragma unroll
                for (int d = 0; d < ND; d++) f[d] = f[d] + pf[d][t - b0];
            }
            __syncwarp();
        }
    }
    if (live) store_force<ND, MODE>(c, i, f);
}

template <int ND, int KIND>
__global__ void __launch_bounds__(F64_THREADS) k_pair64(DevCtx c) {
    forces64<ND, KIND, FM_FORCES, true>(c);
}

// Per-atom sums of the pair forces, one warp per sum64_atoms() atoms on its
// own: in rounds of 32 list entries it gathers the slots of each atom (its own
// pairs are consecutive; another atom's pair is one 32-byte sector), drops the
// zeros and stages the rest in list order, then one lane per (atom, component)
// adds them.  Bound by those FP64 adds and the 32 B per entry from L2 and
// memory: ~30 us of the 114 at 29,667 LJ atoms, 1.0 ms of 3.10 at 1,048,576.
constexpr int SUM64_WARPS = 4;
template <int ND>
constexpr uint32_t sum64_atoms() { return ND == 3 ? 10u : 16u; }   // x ND components: one warp
template <int ND, int MODE>
__global__ void __launch_bounds__(32 * SUM64_WARPS) k_sum64(DevCtx c) {
    constexpr uint32_t ATOMS = sum64_atoms<ND>(), GROUP = ATOMS / 2;
    __shared__ double pf_s[SUM64_WARPS][ND][ATOMS * 33];
    using V = typename SlotVec<ND>::T;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t i0 = (blockIdx.x * SUM64_WARPS + warp) * ATOMS;   // uniform in the warp from here
    if (i0 >= c.n) return;
    double (*pf)[ATOMS * 33] = pf_s[warp];
    // lane a < ATOMS holds atom a's list
    uint32_t nn = 0u, lower = 0u, b0 = 0u;
    bool live = false;
    if (lane < ATOMS && i0 + lane < c.n) {
        const uint32_t i = i0 + lane;
        live = c.active[c.atom_sys[i]] != 0u;
        if (live && c.rank[i] != NOT_MEMBER) {
            nn = c.nnb[i];
            lower = c.half_n[i];
            b0 = c.half_base[i];
        }
    }
    const uint32_t nmax = __reduce_max_sync(0xFFFFFFFFu, nn);
    const uint32_t sa = lane % ATOMS, sd = lane / ATOMS;   // summing lane: atom, component
    double fsum = 0.0;
    for (uint32_t base = 0; base < nmax; base += 32u) {
        const uint32_t k = base + lane;
        uint32_t cnt = 0u;   // lane a: entries staged for atom a
#pragma unroll
        for (uint32_t g = 0; g < 2; g++) {
            V w[GROUP];
            uint32_t second = 0u;   // bit u: the atom is second in the pair
#pragma unroll
            for (uint32_t u = 0; u < GROUP; u++) {   // all loads before any use
                const uint32_t a = g * GROUP + u;
                const uint32_t na = __shfl_sync(0xFFFFFFFFu, nn, a), la = __shfl_sync(0xFFFFFFFFu, lower, a);
                const uint32_t ba = __shfl_sync(0xFFFFFFFFu, b0, a);
                w[u] = V{};
                if (k < na) {
                    const uint32_t sl = k < la ? ba + k : __ldg(c.slots + (size_t)(i0 + a) * c.maxnb + k);
                    if (sl != NO_SLOT) w[u] = static_cast<const V*>(c.pairf)[sl];
                    second |= (k < la ? 0u : 1u) << u;
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < GROUP; u++) {
                const uint32_t a = g * GROUP + u;
                const unsigned long long* wb = reinterpret_cast<const unsigned long long*>(&w[u]);
                unsigned long long any = 0;
#pragma unroll
                for (int d = 0; d < ND; d++) any |= wb[d];
                const uint32_t mask = __ballot_sync(0xFFFFFFFFu, any != 0ull);
                if (any) {
                    const uint32_t q = a * 33u + __popc(mask & ((1u << lane) - 1u));
                    const unsigned long long neg = (unsigned long long)((second >> u) & 1u) << 63;
#pragma unroll
                    for (int d = 0; d < ND; d++) pf[d][q] = __longlong_as_double((long long)(wb[d] ^ neg));
                }
                if (lane == a) cnt = (uint32_t)__popc(mask);
            }
        }
        __syncwarp();
        const uint32_t m = __shfl_sync(0xFFFFFFFFu, cnt, sa);
        if (sd < ND) {
            const double* p = &pf[sd][sa * 33u];
#pragma unroll 4
            for (uint32_t q = 0; q < m; q++) fsum = fsum + p[q];
        }
        __syncwarp();
    }
    // the components of an atom meet in its first staged place
    if (sd < ND) pf[sd][sa * 33u] = fsum;
    __syncwarp();
    if (!live) return;
    double f[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < ND; d++) f[d] = pf[d][lane * 33u];
    store_force<ND, MODE>(c, i0 + lane, f);
}

// per-atom partial sums over the half list (neighbours of smaller rank), i.e.
// each reference pair (first = higher rank) exactly once
template <int ND, int KIND>
__global__ void __launch_bounds__(BLOCK) k_eval64(DevCtx c, int what) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const uint32_t uni = c.uniform;
    const int ncomp = (what == EV_STRESS) ? ND * ND : 1;
    double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const uint32_t ri = c.rank[i];
    if (ri != NOT_MEMBER) {
        const uint32_t s = c.atom_sys[i];
        const SysConst& S = c.sys[s];
        double xi[3] = {0, 0, 0};
        load3<ND>(c.x, i, xi);
        const AtomPrm Pi = c.prm[i];
        const uint32_t nn = c.nnb[i];
        for (uint32_t k = 0; k < nn; k++) {
            const uint32_t j = c.nbr[(size_t)i * c.maxnb + k];
            if (c.rank[j] > ri) continue;
            double xj[3] = {0, 0, 0};
            load3<ND>(c.x, j, xj);
            double r[3] = {0, 0, 0};
            if (S.lees) {
                lees_diff<ND>(S, xi, xj, r);
            } else {
#pragma unroll
                for (int d = 0; d < ND; d++) r[d] = remainder_exact(xi[d] - xj[d], S.L[d], S.invL[d], S.halfL[d]);
            }
            double dsq = r[0] * r[0] + r[1] * r[1];
            if constexpr (ND == 3) dsq = dsq + r[2] * r[2];
            PairC pc;
            if constexpr (idx_kind<KIND>())   // i is the pair's first atom (higher rank)
                pc = combine_idx<KIND>(c, Pi, c.prm[j], __float_as_uint(c.prm32[i].x),
                                       __float_as_uint(c.prm32[j].x), uni);
            else
                pc = combine<KIND>(Pi, c.prm[j], uni);
            if (what == EV_ENERGY || what == EV_CONTACTS || what == EV_OVERLAPS) {
                double e = pair_energy<KIND>(pc, dsq, uni);
                if (what == EV_ENERGY) acc[0] = acc[0] + e;
                else if (what == EV_CONTACTS) acc[0] += (e != 0.0) ? 1.0 : 0.0;
                else acc[0] += (e > 0.0) ? 1.0 : 0.0;
            } else {
                pc.set_derived();   // (the energies do not use these)
                double sc;
                double fo[3] = {0, 0, 0};
                if constexpr (KIND == KIND_REPULSIONDRAG) {
                    double vi[3] = {0, 0, 0}, vj[3] = {0, 0, 0};
                    load3<ND>(c.v, i, vi);
                    load3<ND>(c.v, j, vj);
                    if (!drag_force<ND>(pc, r, dsq, vi, vj, fo))
                        for (int d = 0; d < 3; d++) fo[d] = 0.0;
                } else if (force_scale<KIND>(pc, dsq, uni, sc)) {
#pragma unroll
                    for (int d = 0; d < ND; d++) fo[d] = r[d] * sc;
                }
                if (what == EV_VIRIAL) {
                    double p = r[0] * fo[0] + r[1] * fo[1];
                    if constexpr (ND == 3) p = p + r[2] * fo[2];
                    acc[0] = acc[0] + p;
                } else {
#pragma unroll
                    for (int aa = 0; aa < ND; aa++)
#pragma unroll
                        for (int bb = 0; bb < ND; bb++) acc[aa * ND + bb] = acc[aa * ND + bb] + r[aa] * fo[bb];
                }
            }
        }
    }
    for (int q = 0; q < ncomp; q++) c.red[(size_t)q * c.n + i] = acc[q];
}

template <int ND, int KIND>
static void force64_nd_kind(const DevCtx& c, cudaStream_t s, int mode) {
    const unsigned g = grid_for(c.n, F64_ATOMS);
    if (c.pairf) {
        launch_after(c, k_pair64<ND, KIND>, g, F64_THREADS, 0, s, c);
        const unsigned gs = grid_for(c.n, (int)(SUM64_WARPS * sum64_atoms<ND>()));
        // (not overlapped with k_pair64: its waiting CTAs cost that kernel's tail 5 us at 29,667 atoms)
        if (mode == FM_FORCES_A) k_sum64<ND, FM_FORCES_A><<<gs, 32 * SUM64_WARPS, 0, s>>>(c);
        else k_sum64<ND, FM_FORCES><<<gs, 32 * SUM64_WARPS, 0, s>>>(c);
        return;
    }
    if (c.f64_way == F64_MANY) {
        const unsigned gs = grid_for(c.n, 32 * F64W_WARPS);
        if (mode == FM_FORCES_A) launch_after(c, k_force64w<ND, KIND, FM_FORCES_A>, gs, 32 * F64W_WARPS, 0, s, c);
        else launch_after(c, k_force64w<ND, KIND, FM_FORCES>, gs, 32 * F64W_WARPS, 0, s, c);
        return;
    }
    if (c.f64_way == F64_SHORT) {
        const unsigned gs = grid_for(c.n, F64S_ATOMS);
        if (mode == FM_FORCES_A) launch_after(c, k_force64s<ND, KIND, FM_FORCES_A>, gs, F64S_THREADS, 0, s, c);
        else launch_after(c, k_force64s<ND, KIND, FM_FORCES>, gs, F64S_THREADS, 0, s, c);
        return;
    }
    if (mode == FM_FORCES_A) launch_after(c, k_force64<ND, KIND, FM_FORCES_A>, g, F64_THREADS, 0, s, c);
    else launch_after(c, k_force64<ND, KIND, FM_FORCES>, g, F64_THREADS, 0, s, c);
}

template <int ND>
static void force64_nd(const DevCtx& c, cudaStream_t s, int mode) {
    if (c.kind == KIND_LJCUT) force64_nd_kind<ND, KIND_LJCUT>(c, s, mode);
    else if (c.kind == KIND_LJATTRACT) force64_nd_kind<ND, KIND_LJATTRACT>(c, s, mode);
    else if (c.kind == KIND_LOISOHERN) force64_nd_kind<ND, KIND_LOISOHERN>(c, s, mode);
    else if (c.kind == KIND_LOISLIN) force64_nd_kind<ND, KIND_LOISLIN>(c, s, mode);
    else if (c.kind == KIND_EISMCLACHLAN) force64_nd_kind<ND, KIND_EISMCLACHLAN>(c, s, mode);
    else if (c.kind == KIND_REPULSIONDRAG) force64_nd_kind<ND, KIND_REPULSIONDRAG>(c, s, mode);
    else if (c.kind == KIND_LJCUT_IDX) force64_nd_kind<ND, KIND_LJCUT_IDX>(c, s, mode);
    else if (c.kind == KIND_LJATTRACT_IDX) force64_nd_kind<ND, KIND_LJATTRACT_IDX>(c, s, mode);
    else if (c.kind == KIND_LJATTRACTREPULSE) force64_nd_kind<ND, KIND_LJATTRACTREPULSE>(c, s, mode);
    else if (c.kind == KIND_LJFIXEDREPULSE) force64_nd_kind<ND, KIND_LJFIXEDREPULSE>(c, s, mode);
    else if (c.kind == KIND_LJISH) force64_nd_kind<ND, KIND_LJISH>(c, s, mode);
    else if (c.kind == KIND_REPULSION_IDX) force64_nd_kind<ND, KIND_REPULSION_IDX>(c, s, mode);
    else if (c.kind == KIND_LJATTREPSIGS) force64_nd_kind<ND, KIND_LJATTREPSIGS>(c, s, mode);
    else if (c.kind == KIND_REPULSION) force64_nd_kind<ND, KIND_REPULSION>(c, s, mode);
    else force64_nd_kind<ND, KIND_LJREPULSE>(c, s, mode);
}

void launch_force64(const DevCtx& c, cudaStream_t s, int mode) {
    if (c.nd == 3) force64_nd<3>(c, s, mode); else force64_nd<2>(c, s, mode);
}

template <int ND>
static void eval64_nd(const DevCtx& c, cudaStream_t s, int what) {
    unsigned g = grid_for(c.n);
    if (c.kind == KIND_LJCUT) k_eval64<ND, KIND_LJCUT><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJATTRACT) k_eval64<ND, KIND_LJATTRACT><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LOISOHERN) k_eval64<ND, KIND_LOISOHERN><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LOISLIN) k_eval64<ND, KIND_LOISLIN><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_EISMCLACHLAN) k_eval64<ND, KIND_EISMCLACHLAN><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_REPULSIONDRAG) k_eval64<ND, KIND_REPULSIONDRAG><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJCUT_IDX) k_eval64<ND, KIND_LJCUT_IDX><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJATTRACT_IDX) k_eval64<ND, KIND_LJATTRACT_IDX><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJATTRACTREPULSE) k_eval64<ND, KIND_LJATTRACTREPULSE><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJFIXEDREPULSE) k_eval64<ND, KIND_LJFIXEDREPULSE><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJISH) k_eval64<ND, KIND_LJISH><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_REPULSION_IDX) k_eval64<ND, KIND_REPULSION_IDX><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_LJATTREPSIGS) k_eval64<ND, KIND_LJATTREPSIGS><<<g, BLOCK, 0, s>>>(c, what);
    else if (c.kind == KIND_REPULSION) k_eval64<ND, KIND_REPULSION><<<g, BLOCK, 0, s>>>(c, what);
    else k_eval64<ND, KIND_LJREPULSE><<<g, BLOCK, 0, s>>>(c, what);
}

void launch_eval64(const DevCtx& c, cudaStream_t s, int what) {
    if (c.nd == 3) eval64_nd<3>(c, s, what); else eval64_nd<2>(c, s, what);
}

}  // namespace parm
