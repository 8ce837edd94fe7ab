// Mixed-precision cell-block kernels: list build, pair forces and list
// expansion with the neighbourhood of a block of cells staged in shared memory
// (blocks, staged records and lists: staged.cuh).
#include <algorithm>

#include "staged.cuh"

namespace parm {

// ---------------------------------------------------------------------------
// list build: one CTA per block, one thread per home atom
// ---------------------------------------------------------------------------
// plain position of local index q; w: the list diameter (DIA) or 0
template <int ND, int DIA>
__device__ __forceinline__ float4 stg_get_plain(const DevCtx& c, const SysConst& S, const StgTable& T,
                                                const float4* sp, uint32_t cap, uint32_t q) {
    if (q < cap) return stg_at_plain(sp, q);
    const uint32_t p = stg_piece(T, q);
    const uint32_t j = T.g0[p] + (q - T.off[p]);
    return stg_plain(T, stg_shift(T, p, c.rec[j]), DIA ? stg_diam(c, j) : 0.f);
}

template <int ND, int DIA, bool FULL>
__device__ __forceinline__ void build_home(const DevCtx& c, const SysConst& S, const StgTable& T,
                                           const float4* sp, uint32_t cap, const HomeAtom& a) {
    const uint32_t maxnb = c.maxnb;
    uint16_t* out = c.nbr16;
    const float skin32 = (float)S.skin;
    const float4 P = FULL ? stg_at_plain(sp, a.qi) : stg_get_plain<ND, DIA>(c, S, T, sp, cap, a.qi);
    const float tu = (DIA ? P.w : stg_diam(c, a.i)) + skin32;
    const float hiu = tu * tu * (1.0f + STG_BAND), lou = tu * tu * (1.0f - STG_BAND);
    const uint32_t oi = c.excl_off ? c.orig[a.i] : 0u;
    // entry k of this atom: ob[(k / 2) * 2H + k % 2], i.e. half k % 2 of the
    // 32-bit word ow[(k / 2) * H] (maxnb is a multiple of 8)
    uint16_t* const ob = out + (size_t)a.s0 * maxnb + 2u * a.hs;
    uint32_t* const ow = reinterpret_cast<uint32_t*>(ob);
    const uint32_t H2 = 2u * a.H;
    uint32_t k = 0, pend = 0u;
    // broadcast pairs for the packed screening of FULL stages
    const f32x2 Px2 = pk2(P.x, P.x), Py2 = pk2(P.y, P.y), Pz2 = pk2(P.z, P.z);
    const f32x2 HI2 = pk2(hiu, hiu), LO2 = pk2(lou, lou);
    const f32x2 PW2 = pk2(P.w, P.w), HALF2 = pk2(0.5f, 0.5f), SKIN2 = pk2(skin32, skin32);
    const f32x2 BH2 = pk2(1.0f + STG_BAND, 1.0f + STG_BAND), BL2 = pk2(1.0f - STG_BAND, 1.0f - STG_BAND);
#pragma unroll 1
    for (int dz = 0; dz < (ND == 3 ? 3 : 1); dz++) {
#pragma unroll 1
        for (int dy = 0; dy < 3; dy++) {
            const uint32_t r = (uint32_t)dz * T.nyr + a.hr + (uint32_t)dy;
            uint32_t lo, hi;
            stg_range(c, T, r, a.cx, lo, hi);
            // 32 candidates at a time: a branch-free screening pass sets one
            // bit per candidate within the widened threshold, then the set
            // bits (the ~15 % that are kept) are settled and written in order
#pragma unroll 1
            // FULL stages are screened two candidates at a time in packed
            // FP32 pairs, so the passes start at an even local index (an odd
            // row start adds the slot before it, cleared below)
            for (uint32_t base = FULL ? (lo & ~1u) : lo; base < hi; base += 32u) {
                const uint32_t m = min(32u, hi - base);
                uint32_t mask = 0u, sure = 0u;
                // bit of a candidate within the widened threshold (mask) and
                // within the narrowed one (sure: kept without the exact test)
                auto screen = [&](const float4& Q, uint32_t bit) {
                    const float dx = P.x - Q.x, dyv = P.y - Q.y;
                    float rr = fmaf(dyv, dyv, dx * dx);
                    if constexpr (ND == 3) {
                        const float dzv = P.z - Q.z;
                        rr = fmaf(dzv, dzv, rr);
                    }
                    float hi2 = hiu, lo2 = lou;
                    if constexpr (DIA) {
                        const float thr = 0.5f * (P.w + Q.w) + skin32;
                        hi2 = thr * thr * (1.0f + STG_BAND);
                        lo2 = thr * thr * (1.0f - STG_BAND);
                    }
                    mask |= rr <= hi2 ? bit : 0u;
                    sure |= rr < lo2 ? bit : 0u;
                };
                if constexpr (FULL) {
                    // all 32 slots (the stage has 32 records of padding past
                    // its capacity), then the slots past the row, the slot
                    // before an odd row start and the home atom itself are
                    // cleared.  A candidate's bit is the sign of rr - hi2
                    // (rr < hi2; equality is far outside the true threshold,
                    // which lies 2e-5 below hi2) and of rr - lo2 (rr < lo2),
                    // shifted in from the top candidate down so that bit u
                    // is candidate base + u.
                    const ulonglong2* sq = reinterpret_cast<const ulonglong2*>(sp) + base;
#pragma unroll
                    for (int u2 = 15; u2 >= 0; u2--) {
                        const ulonglong2 A = sq[2 * u2];   // (x0, x1), (y0, y1)
                        const f32x2 dx = sub2(Px2, A.x), dy = sub2(Py2, A.y);
                        f32x2 rr = fma2(dy, dy, mul2(dx, dx));
                        f32x2 h2 = HI2, l2 = LO2;
                        if constexpr (ND == 3 || DIA) {
                            const ulonglong2 B = sq[2 * u2 + 1];   // (z0, z1), (w0, w1)
                            if constexpr (ND == 3) {
                                const f32x2 dz = sub2(Pz2, B.x);
                                rr = fma2(dz, dz, rr);
                            }
                            if constexpr (DIA) {
                                const f32x2 thr = fma2(add2(PW2, B.y), HALF2, SKIN2);
                                const f32x2 t2 = mul2(thr, thr);
                                h2 = mul2(t2, BH2);
                                l2 = mul2(t2, BL2);
                            }
                        }
                        float e0, e1, g0, g1;
                        upk2(sub2(rr, h2), e0, e1);
                        upk2(sub2(rr, l2), g0, g1);
                        mask = __funnelshift_l(__float_as_uint(e1), mask, 1);
                        sure = __funnelshift_l(__float_as_uint(g1), sure, 1);
                        mask = __funnelshift_l(__float_as_uint(e0), mask, 1);
                        sure = __funnelshift_l(__float_as_uint(g0), sure, 1);
                    }
                    if (m < 32u) mask &= (1u << m) - 1u;
                    if (base < lo) mask &= ~1u;
                    const uint32_t d = a.qi - base;
                    if (d < 32u) mask &= ~(1u << d);
                } else {
#pragma unroll 8
                    for (uint32_t u = 0; u < m; u++) {
                        const uint32_t q = base + u;
                        if (q != a.qi) screen(stg_get_plain<ND, DIA>(c, S, T, sp, cap, q), 1u << u);
                    }
                }
                // entries are written as 32-bit words of two (the even one
                // waits in `pend`)
                if ((mask & ~sure) == 0u && !c.excl_off) {
                    while (mask) {   // all kept
                        const uint32_t q = base + (uint32_t)__ffs(mask) - 1u;
                        mask &= mask - 1u;
                        if (k < maxnb) {
                            if (k & 1u) ow[(size_t)(k >> 1) * a.H] = pend | (q << 16);
                            else pend = q;
                        }
                        k++;
                    }
                    continue;
                }
                while (mask) {
                    const uint32_t u = (uint32_t)__ffs(mask) - 1u;
                    mask &= mask - 1u;
                    const uint32_t q = base + u;
                    bool keep = (sure >> u) & 1u;
                    uint32_t j = 0xFFFFFFFFu;
                    if (!keep) {   // rare: the exact reference test
                        j = stg_global(T, q);
                        keep = keep_exact_rn<ND>(c, S, a.i, j);
                    }
                    if (keep && c.excl_off) {
                        if (j == 0xFFFFFFFFu) j = stg_global(T, q);
                        keep = !is_excluded_s(c, oi, c.orig[j]);
                    }
                    if (!keep) continue;
                    if (k < maxnb) {
                        if (k & 1u) ow[(size_t)(k >> 1) * a.H] = pend | (q << 16);
                        else pend = q;
                    }
                    k++;
                }
            }
        }
    }
    {
        const uint32_t kk = min(k, maxnb);
        if (kk & 1u) ob[(size_t)(kk >> 1) * H2] = (uint16_t)pend;   // the last, unpaired entry
    }
    if (k > maxnb) {
        atomicOr(c.status, ST_NBR_OVERFLOW);
        k = maxnb;
    }
    c.nnb[a.i] = k;
    atomicMax(const_cast<uint32_t*>(&T.hnmax[a.hr]), k);
}

template <int ND, int DIA>
__global__ void __launch_bounds__(STG_THREADS, 4) k_build_stg(DevCtx c) {
    extern __shared__ float4 smem_b[];
    __shared__ StgTable T;
    if (blockIdx.x >= c.nblk) {
        const uint32_t s = blockIdx.x - c.nblk;
        if (c.flag[s]) stg_nonmembers(c, s, 0);
        return;
    }
    const uint4 bd = c.blk[blockIdx.x];
    if (!c.flag[bd.x]) return;
    const SysConst& S = c.sys[bd.x];
    stg_setup<ND>(c, S, bd, T);
    stg_prefetch<ND>(c, T, false);
    if (T.total > 0xFFFFu) {   // more than 65535 atoms around one block
        if (threadIdx.x == 0) atomicOr(c.status, ST_TILE_OVERFLOW);
        return;
    }
    const uint32_t cap = c.stg_cap;
    stg_load_plain(c, T, smem_b, cap, DIA != 0);
    const bool full = T.total <= cap;
    for (uint32_t h = threadIdx.x; h < T.nhome; h += blockDim.x) {
        const HomeAtom a = stg_home<ND>(c, T, h);
        if (full) build_home<ND, DIA, true>(c, S, T, smem_b, cap, a);
        else build_home<ND, DIA, false>(c, S, T, smem_b, cap, a);
    }
    __syncthreads();   // the home rows' longest lists are in the table now
    stg_store_table(c, T, blockIdx.x);
}

// ---------------------------------------------------------------------------
// pair forces: one CTA per block, one thread per home atom.  PRM: 0 uniform
// parameters, 1 per-atom sigma (epsilon and exponent / cut-off uniform),
// 2 per-atom (sqrt(eps), sigma, third).  A launch loads the block's table
// (stored by the list build), requests the pieces' records and the used part
// of the home rows' lists into L2, copies the records into shared memory with
// one bulk asynchronous copy per piece and moves them into the block frame.
// ---------------------------------------------------------------------------
// pair-law constants of one pair type
template <int KIND>
struct Law {
    float e12, isig2, sig, third, C, cut2, band;
    __device__ __forceinline__ void set(float e12_, float sig_, float isig2_, float third_) {
        e12 = e12_;
        sig = sig_;
        isig2 = isig2_;
        third = third_;
        C = e12 * isig2;
        cut2 = (KIND == KIND_LJCUT) ? third * third : 1.0f;
        band = CUT_BAND_S * cut2;
    }
    // LJ kinds: the force scale s (F_i += r * s) ignoring the cut-off, and
    // dd = r^2/sigma^2 - cut^2
    __device__ __forceinline__ float lj_raw(float d2, float& dd) const {
        const float rsq = d2 * isig2;
        const float ir = rcp_approx(rsq);
        const float ir2 = ir * ir;
        const float ir4 = ir2 * ir2;
        const float ir3 = ir2 * ir;
        const float t = C * ir4;
        dd = rsq - cut2;
        return fmaf(t, ir3, -t);   // 12 eps / sigma^2 * ir^4 (ir^3 - 1)
    }
    // force scale s (F_i += r * s), zero beyond the FP32 cut-off test; for
    // LJCUT, `dmin` tracks min(|dd| - band): a pair with |dd| <= band is
    // settled afterwards by the exact FP64 test
    __device__ __forceinline__ float scale(float d2, float& dmin) const {
        if constexpr (KIND == KIND_LJCUT || KIND == KIND_LJREPULSE) {
            float dd;
            const float sc = lj_raw(d2, dd);
            if constexpr (KIND == KIND_LJCUT) dmin = fminf(dmin, fabsf(dd) - band);
            return dd > 0.0f ? 0.0f : sc;
        } else {
            bool nc;
            return scale32<KIND>(d2, e12, sig, isig2, third, nc);
        }
    }
};

// per-home-atom data loaded from global memory before the pair loop (issued
// ahead of the staging wait for a thread's first home atom)
struct HomePre {
    uint32_t nn, w0, w1;
    float4 Qi;   // (sqrt(eps), sigma, third, m6)
    const uint32_t* row;
};

// MULTI: thread `sub` of 2^lg takes the words sub, sub + 2^lg, ...
template <bool MULTI = false>
__device__ __forceinline__ HomePre home_pre(const DevCtx& c, const HomeAtom& a, uint32_t sub = 0u, uint32_t lg = 0u) {
    HomePre p;
    p.nn = c.nnb[a.i];
    p.Qi = c.prm32[a.i];
    p.row = reinterpret_cast<const uint32_t*>(c.nbr16) + ((size_t)a.s0 * c.maxnb >> 1) + a.hs;
    if constexpr (MULTI) {
        p.row += (size_t)sub * a.H;
        const uint32_t nw = (p.nn + 1u) >> 1;   // words in use
        p.w0 = sub < nw ? __ldg(p.row) : 0u;
        p.w1 = sub + (1u << lg) < nw ? __ldg(p.row + ((size_t)a.H << lg)) : 0u;
        return p;
    }
    p.w0 = __ldg(p.row);       // entries of the first two words (read even when
    p.w1 = __ldg(p.row + a.H); // the list is shorter: they lie inside its region)
    return p;
}

template <int ND, int KIND, int PRM, bool FULL, bool MULTI>
__device__ __forceinline__ void force_home(const DevCtx& c, const SysConst& S, const StgTable& T,
                                           const float4* srec, const void* sext, uint32_t cap,
                                           const HomeAtom& a, const HomePre& pre, const Law<KIND>& law0,
                                           float* f, uint32_t hidx, uint32_t sub, uint32_t lg) {
    float dmin = 1.0f;   // min over pairs of |rsq - cut^2| - band (LJCUT)
    const float4 ri = FULL ? srec[a.qi] : stg_get<ND>(c, S, T, srec, cap, a.qi);
    const uint32_t wi = stg_wi(ri);
    const float* ssig = static_cast<const float*>(sext);
    const float4* sprm = static_cast<const float4*>(sext);
    const float4 Qi = pre.Qi;
    // MULTI: this thread's words, as a list of its own (every word's entries but
    // the high half of the list's last word when its length is odd)
    uint32_t nn = pre.nn, H = a.H;
    if constexpr (MULTI) {
        const uint32_t nw = (nn + 1u) >> 1, split = 1u << lg;
        const uint32_t mine = nw > sub ? (nw - sub + split - 1u) >> lg : 0u;
        const bool last = mine && sub + ((mine - 1u) << lg) == nw - 1u;
        nn = 2u * mine - ((last && (nn & 1u)) ? 1u : 0u);
        H <<= lg;
    }
    const uint32_t* row = pre.row;
    const uint32_t qmax = T.total - 1u;
    auto pair = [&](uint32_t q) {
        float4 rj;
        if (FULL) {
            q = min(q, qmax);
            rj = srec[q];
        } else {
            q = stg_check(c, T, q, a.qi);
            if (q == a.qi) return;
            rj = stg_get<ND>(c, S, T, srec, cap, q);
        }
        float r[3];
        stg_disp<ND>(wi, ri, rj, r);
        float d2 = fmaf(r[1], r[1], r[0] * r[0]);
        if constexpr (ND == 3) d2 = fmaf(r[2], r[2], d2);
        Law<KIND> law = law0;
        if constexpr (PRM == 1) {
            const float sj = (FULL || q < cap) ? ssig[q] : c.prm32[stg_global(T, q)].y;
            const float sg = 0.5f * (Qi.y + sj);
            law.set(law0.e12, sg, rcp_approx(sg * sg), law0.third);
        } else if constexpr (PRM == 2) {
            const float4 Qj = (FULL || q < cap) ? sprm[q] : c.prm32[stg_global(T, q)];
            const float eps = Qi.x * Qj.x;
            const float sg = 0.5f * (Qi.y + Qj.y);
            law.set((KIND == KIND_REPULSION) ? eps : 12.0f * eps, sg, rcp_approx(sg * sg),
                    (KIND == KIND_LJCUT) ? fmaxf(Qi.z, Qj.z) : 0.5f * (Qi.z + Qj.z));
        }
        const float sc = law.scale(d2, dmin);
#pragma unroll
        for (int d = 0; d < ND; d++) f[d] = fmaf(r[d], sc, f[d]);
    };
    const uint32_t nw = nn >> 1;   // words holding two entries
    uint32_t p = 0;
    if constexpr (FULL && PRM == 0 && (KIND == KIND_LJCUT || KIND == KIND_LJREPULSE)) {
        // the two entries of each list word together, in packed FP32 pairs:
        // even entries accumulate in the low half, odd ones in the high half
        const f32x2 K2 = pk2(STG_K, STG_K), is2 = pk2(law0.isig2, law0.isig2), C2 = pk2(law0.C, law0.C);
        const f32x2 P1_2 = pk2(1.0f, 1.0f);
        f32x2 fx = pk2(0.f, 0.f), fy = fx, fz = fx;
        auto pair2 = [&](uint32_t w) {
            const uint32_t q0 = min(w & 0xFFFFu, qmax), q1 = min(w >> 16, qmax);
            const float4 ra = srec[q0], rb = srec[q1];
            const uint32_t D0 = wi - __float_as_uint(ra.w), D1 = wi - __float_as_uint(rb.w);
            const f32x2 rx = add2(sub2(pk2(__uint_as_float((D0 & 0xFFFu) | STG_MANT),
                                           __uint_as_float((D1 & 0xFFFu) | STG_MANT)), K2),
                                  pk2(ri.x - ra.x, ri.x - rb.x));
            const f32x2 ry = add2(sub2(pk2(__uint_as_float(((D0 >> 12) & 0x3FFu) | STG_MANT),
                                           __uint_as_float(((D1 >> 12) & 0x3FFu) | STG_MANT)), K2),
                                  pk2(ri.y - ra.y, ri.y - rb.y));
            f32x2 d2 = fma2(ry, ry, mul2(rx, rx));
            f32x2 rz = pk2(0.f, 0.f);
            if constexpr (ND == 3) {
                rz = add2(sub2(pk2(__uint_as_float((D0 >> 22) | STG_MANT), __uint_as_float((D1 >> 22) | STG_MANT)),
                               K2),
                          pk2(ri.z - ra.z, ri.z - rb.z));
                d2 = fma2(rz, rz, d2);
            }
            float r0, r1;
            upk2(mul2(d2, is2), r0, r1);
            const f32x2 ir = pk2(rcp_approx(r0), rcp_approx(r1));
            const f32x2 ir2 = mul2(ir, ir);
            const f32x2 ir4 = mul2(ir2, ir2);
            const f32x2 ir3 = mul2(ir2, ir);
            const f32x2 t = mul2(C2, ir4);
            float s0, s1;
            // 12 eps / sigma^2 * ir^4 (ir^3 - 1); ir^3 - 1 is exact for ir^3 in
            // [1/2, 2] (the strongly repulsive and the attractive well's pairs),
            // so the product is the only rounding there
            upk2(mul2(t, sub2(ir3, P1_2)), s0, s1);
            const float dd0 = r0 - law0.cut2, dd1 = r1 - law0.cut2;
            if constexpr (KIND == KIND_LJCUT) dmin = fminf(dmin, fminf(fabsf(dd0), fabsf(dd1)) - law0.band);
            const f32x2 sc = pk2(dd0 > 0.0f ? 0.0f : s0, dd1 > 0.0f ? 0.0f : s1);
            fx = fma2(rx, sc, fx);
            fy = fma2(ry, sc, fy);
            if constexpr (ND == 3) fz = fma2(rz, sc, fz);
        };
        if (nw >= 2) {
            uint32_t w0 = pre.w0, w1 = pre.w1;
#pragma unroll 1
            for (; p + 3 < nw; p += 2) {
                const uint32_t n0 = __ldg(row + (size_t)(p + 2) * H), n1 = __ldg(row + (size_t)(p + 3) * H);
                pair2(w0);
                pair2(w1);
                w0 = n0;
                w1 = n1;
            }
            pair2(w0);
            pair2(w1);
            p += 2;
        }
        if (p < nw) pair2(p == 0 ? pre.w0 : __ldg(row + (size_t)p * H));
        float a0, a1;
        upk2(fx, a0, a1);
        f[0] = a0 + a1;
        upk2(fy, a0, a1);
        f[1] = a0 + a1;
        if constexpr (ND == 3) {
            upk2(fz, a0, a1);
            f[2] = a0 + a1;
        }
        p = nw;
    }
    if (nw >= 2 && p == 0) {
        uint32_t w0 = pre.w0, w1 = pre.w1;
#pragma unroll 1
        for (; p + 3 < nw; p += 2) {
            const uint32_t n0 = __ldg(row + (size_t)(p + 2) * H), n1 = __ldg(row + (size_t)(p + 3) * H);
            pair(w0 & 0xFFFFu);
            pair(w0 >> 16);
            pair(w1 & 0xFFFFu);
            pair(w1 >> 16);
            w0 = n0;
            w1 = n1;
        }
        pair(w0 & 0xFFFFu);
        pair(w0 >> 16);
        pair(w1 & 0xFFFFu);
        pair(w1 >> 16);
        p += 2;
    }
    if (p < nw) {
        const uint32_t w = p == 0 ? pre.w0 : __ldg(row + (size_t)p * H);
        pair(w & 0xFFFFu);
        pair(w >> 16);
    }
    if (nn & 1u) pair((nw == 0 ? pre.w0 : (nw == 1 ? pre.w1 : __ldg(row + (size_t)nw * H))) & 0xFFFFu);
    if constexpr (MULTI) {
        // the atom's threads are neighbouring lanes of one warp
        const uint32_t lane = threadIdx.x & 31u, split = 1u << lg;
        const uint32_t group = (split == 32u ? 0xFFFFFFFFu : (1u << split) - 1u) << (lane & ~(split - 1u));
        for (uint32_t o = split >> 1; o; o >>= 1) {
#pragma unroll
            for (int d = 0; d < ND; d++) f[d] += __shfl_xor_sync(group, f[d], o);
            if constexpr (KIND == KIND_LJCUT) dmin = fminf(dmin, __shfl_xor_sync(group, dmin, o));
        }
        if (sub) return;
    }
    if constexpr (KIND == KIND_LJCUT) {
        // rare: a pair within the cut-off band; k_band_stg settles it by the
        // exact FP64 test after this kernel (kept out of this loop so that the
        // loop keeps its registers)
        if (dmin <= 0.0f) {
            const uint32_t k = atomicAdd(c.bandn, 1u);
            if (k < c.n) c.bandq[k] = make_uint2(blockIdx.x, hidx);
        }
    }
}

// MULTI: 2^stg_lg threads per home atom (small systems: blocks with few home
// atoms, so that there are blocks for every SM, and short serial lists)
template <int ND, int KIND, int MODE, int PRM, bool MULTI>
__global__ void __launch_bounds__(STG_THREADS, 5) k_force_stg(DevCtx c) {
    extern __shared__ float4 smem_f[];
    __shared__ StgTable T;
    // until wait_previous() only what list builds and uploads set is read
    // (never what the drift before writes), and nothing is written
    release_next();
    if (blockIdx.x >= c.nblk) {
        wait_previous();
        if (c.active[blockIdx.x - c.nblk]) stg_nonmembers(c, blockIdx.x - c.nblk, MODE == FM_FORCES_A);
        return;
    }
    const uint4 bd = c.blk[blockIdx.x];
    if (!c.active[bd.x]) return;   // frozen system: forces unchanged
    const SysConst& S = c.sys[bd.x];
    stg_load_table(c, T, blockIdx.x);
    stg_prefetch<ND>(c, T, true);   // (into L2, where the drift's writes land too)
    const uint32_t cap = c.stg_cap;
    float4* srec = smem_f;
    void* sext = smem_f + cap;
    // the first home atom's global data is requested before the staging
    // wait, so its latency overlaps with the bulk copies
    HomeAtom a0{};
    HomePre p0{};
    const uint32_t lg = MULTI ? c.stg_lg : 0u, sub = MULTI ? threadIdx.x & ((1u << lg) - 1u) : 0u;
    const uint32_t hfirst = MULTI ? threadIdx.x >> lg : threadIdx.x;
    const bool has0 = hfirst < T.nhome;
    if (has0) {
        a0 = stg_home<ND, false>(c, T, hfirst);
        p0 = home_pre<MULTI>(c, a0, sub, lg);
    }
    __shared__ uint64_t bar;
    wait_previous();
    if (!stg_load_bulk<ND, PRM>(c, T, srec, sext, cap, &bar)) return;
    const bool full = T.total <= cap;
    for (uint32_t h = hfirst; h < T.nhome; h += MULTI ? blockDim.x >> lg : blockDim.x) {
        const HomeAtom a = h == hfirst ? a0 : stg_home<ND, false>(c, T, h);
        const HomePre pre = h == hfirst ? p0 : home_pre<MULTI>(c, a, sub, lg);
        const float4 Qi = pre.Qi;
        Law<KIND> law;
        law.set((KIND == KIND_REPULSION) ? Qi.x * Qi.x : 12.0f * Qi.x * Qi.x, Qi.y, rcp_approx(Qi.y * Qi.y),
                Qi.z);
        float f[3] = {0.f, 0.f, 0.f};
        if (full) force_home<ND, KIND, PRM, true, MULTI>(c, S, T, srec, sext, cap, a, pre, law, f, h, sub, lg);
        else force_home<ND, KIND, PRM, false, MULTI>(c, S, T, srec, sext, cap, a, pre, law, f, h, sub, lg);
        if (MULTI && sub) continue;
        c.f32[a.i] = make_float4(f[0], f[1], f[2], 0.f);
        if constexpr (MODE == FM_FORCES_A) {
            using V = typename DVec<ND>::T;
            V av;
            double* ad = reinterpret_cast<double*>(&av);
#pragma unroll
            for (int d = 0; d < (int)(sizeof(V) / 8); d++) ad[d] = 0.0;
            const double m = c.m[a.i];
            if (!(m <= 0.0 || isinf(m))) {
                const float im = c.invm32[a.i];
#pragma unroll
                for (int d = 0; d < ND; d++) ad[d] = (double)(f[d] * im);
            }
            static_cast<V*>(c.a)[a.i] = av;
        }
    }
}

// Settles the home atoms that k_force_stg listed as having a pair within the
// LJ cut-off band: their force is the kernel's FP32 sum plus the exact-test
// corrections, added in list order as if done inline (records are rebuilt
// from global memory, identical to the staged ones).  One CTA of BAND_WARPS
// warps per listed atom: warp w tests the list's chunks w, w + BAND_WARPS,
// ... of 32 entries in parallel (each lane one entry), the corrections are
// collected per entry and one thread adds them in list order.
constexpr uint32_t BAND_WARPS = 3;
constexpr uint32_t BAND_MAXK = 512;   // longer lists: the corrections of one chunk at a time

template <int ND, int KIND, int MODE, int PRM>
__global__ void __launch_bounds__(32 * BAND_WARPS) k_band_stg(DevCtx c) {
    __shared__ StgTable T;
    __shared__ float4 corr[BAND_MAXK];
    __shared__ uint32_t flags[BAND_MAXK / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    wait_previous();
    const uint32_t nb = min(*c.bandn, c.n);
    for (uint32_t it_k = blockIdx.x; it_k < nb; it_k += gridDim.x) {
        const uint2 it = c.bandq[it_k];
        const uint4 bd = c.blk[it.x];
        const SysConst& S = c.sys[bd.x];
        stg_load_table(c, T, it.x);
        const HomeAtom a = stg_home<ND, false>(c, T, it.y);
        const HomePre pre = home_pre(c, a);
        const float4 Qi = pre.Qi;
        const float4 ri = stg_get<ND>(c, S, T, nullptr, 0u, a.qi);
        const uint32_t wi = stg_wi(ri);
        Law<KIND> law0;
        law0.set(12.0f * Qi.x * Qi.x, Qi.y, rcp_approx(Qi.y * Qi.y), Qi.z);
        // the correction of entry k (FP32 pair force kept or cut wrongly)
        auto entry = [&](uint32_t k, float* cv) -> bool {
            const uint32_t w = __ldg(pre.row + (size_t)(k >> 1) * a.H);
            const uint32_t q = stg_check(c, T, (k & 1u) ? (w >> 16) : (w & 0xFFFFu), a.qi);
            if (q == a.qi) return false;
            const float4 rj = stg_get<ND>(c, S, T, nullptr, 0u, q);
            float r[3];
            stg_disp<ND>(wi, ri, rj, r);
            float d2 = fmaf(r[1], r[1], r[0] * r[0]);
            if constexpr (ND == 3) d2 = fmaf(r[2], r[2], d2);
            Law<KIND> law = law0;
            if constexpr (PRM == 1) {
                const float sg = 0.5f * (Qi.y + c.prm32[stg_global(T, q)].y);
                law.set(law0.e12, sg, rcp_approx(sg * sg), law0.third);
            } else if constexpr (PRM == 2) {
                const float4 Qj = c.prm32[stg_global(T, q)];
                const float sg = 0.5f * (Qi.y + Qj.y);
                law.set(12.0f * Qi.x * Qj.x, sg, rcp_approx(sg * sg), fmaxf(Qi.z, Qj.z));
            }
            float dd;
            const float sc = law.lj_raw(d2, dd);
            if (fabsf(dd) > law.band) return false;
            const bool beyond = lj_beyond_exact_s(c, S, a.i, stg_global(T, q), ND);
            if (beyond == (dd > 0.0f)) return false;   // the FP32 test agreed
            const float sg = beyond ? -sc : sc;
#pragma unroll
            for (int d = 0; d < 3; d++) cv[d] = d < ND ? r[d] * sg : 0.f;
            return true;
        };
        const float4 f0 = c.f32[a.i];
        float f[3] = {f0.x, f0.y, f0.z};
        if (pre.nn <= BAND_MAXK) {
            for (uint32_t t = threadIdx.x; t < BAND_MAXK / 32; t += blockDim.x) flags[t] = 0u;
            __syncthreads();
            for (uint32_t base = 32u * warp; base < pre.nn; base += 32u * BAND_WARPS) {
                const uint32_t k = base + lane;
                float cv[3];
                if (k < pre.nn && entry(k, cv)) {
                    corr[k] = make_float4(cv[0], cv[1], cv[2], 0.f);
                    atomicOr(&flags[k >> 5], 1u << (k & 31u));
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                for (uint32_t wd = 0; wd < (pre.nn + 31u) / 32u; wd++) {
                    uint32_t m = flags[wd];
                    while (m) {
                        const uint32_t k = 32u * wd + (uint32_t)__ffs(m) - 1u;
                        m &= m - 1u;
                        const float4 v = corr[k];
                        f[0] += v.x;
                        f[1] += v.y;
                        f[2] += v.z;
                    }
                }
            }
        } else if (warp == 0) {
            // very long list: one warp, one chunk at a time, in list order
            for (uint32_t base = 0; base < pre.nn; base += 32u) {
                const uint32_t k = base + lane;
                float cv[3] = {0.f, 0.f, 0.f};
                const bool need = k < pre.nn && entry(k, cv);
                uint32_t mask = __ballot_sync(0xFFFFFFFFu, need);
                while (mask) {
                    const int src = __ffs(mask) - 1;
                    mask &= mask - 1u;
#pragma unroll
                    for (int d = 0; d < 3; d++) f[d] += __shfl_sync(0xFFFFFFFFu, cv[d], src);
                }
            }
        }
        if (threadIdx.x == 0) {
            c.f32[a.i] = make_float4(f[0], f[1], f[2], 0.f);
            if constexpr (MODE == FM_FORCES_A) {
                const double m = c.m[a.i];
                if (!(m <= 0.0 || isinf(m))) {
                    const float im = c.invm32[a.i];
                    double* ad = static_cast<double*>(c.a) + (size_t)a.i * (ND == 3 ? 4 : 2);
                    ad[0] = (double)(f[0] * im);
                    ad[1] = (double)(f[1] * im);
                    if constexpr (ND == 3) ad[2] = (double)(f[2] * im);
                }
            }
        }
        __syncthreads();
    }
    if (last_block(&c.done[0], gridDim.x) && threadIdx.x == 0) *c.bandn = 0u;   // for the next force launch
}

// ---------------------------------------------------------------------------
// expansion of the staged lists into the row-major global-index lists used by
// the evaluation kernels and the pair listing (same pairs, same order)
// ---------------------------------------------------------------------------
template <int ND>
__global__ void __launch_bounds__(STG_THREADS) k_expand_stg(DevCtx c) {
    __shared__ StgTable T;
    if (blockIdx.x >= c.nblk) return;
    const uint4 bd = c.blk[blockIdx.x];
    const SysConst& S = c.sys[bd.x];
    stg_setup<ND>(c, S, bd, T);
    const uint32_t maxnb = c.maxnb;
    for (uint32_t h = threadIdx.x; h < T.nhome; h += blockDim.x) {
        const HomeAtom a = stg_home<ND>(c, T, h);
        const uint32_t nn = c.nnb[a.i];
        for (uint32_t k = 0; k < nn; k++)
            c.nbr[(size_t)a.i * maxnb + k] = stg_global(T, stg_check(c, T, c.nbr16[stg_entry16(a, maxnb, k)], a.qi));
    }
}

// the inverse: row-major lists (global indices, built on the same cell grid)
// -> staged lists; every neighbour lies in one of the home atom's stencil rows
template <int ND>
__global__ void __launch_bounds__(STG_THREADS) k_compress_stg(DevCtx c) {
    __shared__ StgTable T;
    if (blockIdx.x >= c.nblk) return;
    const uint4 bd = c.blk[blockIdx.x];
    const SysConst& S = c.sys[bd.x];
    stg_setup<ND>(c, S, bd, T);
    const uint32_t maxnb = c.maxnb;
    for (uint32_t h = threadIdx.x; h < T.nhome; h += blockDim.x) {
        const HomeAtom a = stg_home<ND>(c, T, h);
        const uint32_t nn = c.nnb[a.i];
        for (uint32_t k = 0; k < nn; k++) {
            const uint32_t j = c.nbr[(size_t)a.i * maxnb + k];
            uint32_t q = 0xFFFFFFFFu;
            for (uint32_t p = 0; p < T.npiece; p++)
                if (j - T.g0[p] < T.cnt[p]) {
                    q = T.off[p] + (j - T.g0[p]);
                    break;
                }
            if (q > 0xFFFFu) {
                atomicOr(c.status, ST_TILE_OVERFLOW);
                q = a.qi;
            }
            c.nbr16[stg_entry16(a, maxnb, k)] = (uint16_t)q;
        }
    }
    __syncthreads();
    stg_row_nmax<ND>(c, T);
    stg_store_table(c, T, blockIdx.x);
}

// ---------------------------------------------------------------------------
// the list build reads up to 31 records past a row's end: 32 records of padding
static size_t stg_smem_build(const DevCtx& c) { return ((size_t)c.stg_cap + 32) * sizeof(float4); }
static size_t stg_smem_force(const DevCtx& c) {
    const size_t ext = c.stg_prm == 1 ? sizeof(float) : (c.stg_prm == 2 ? sizeof(float4) : 0);
    return (size_t)c.stg_cap * (sizeof(float4) + ext);
}

template <class K>
static void set_smem(K kern, size_t bytes) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <int ND, int KIND, int MODE>
static void limits_prm(size_t sm) {
    set_smem(k_force_stg<ND, KIND, MODE, 0, false>, sm);
    set_smem(k_force_stg<ND, KIND, MODE, 1, false>, sm);
    set_smem(k_force_stg<ND, KIND, MODE, 2, false>, sm);
    set_smem(k_force_stg<ND, KIND, MODE, 0, true>, sm);
    set_smem(k_force_stg<ND, KIND, MODE, 1, true>, sm);
    set_smem(k_force_stg<ND, KIND, MODE, 2, true>, sm);
}
template <int ND, int KIND>
static void limits_kind(size_t sm) {
    limits_prm<ND, KIND, FM_FORCES>(sm);
    limits_prm<ND, KIND, FM_FORCES_A>(sm);
}
template <int ND>
static void limits_nd(size_t build, size_t force) {
    set_smem(k_build_stg<ND, 0>, build);
    set_smem(k_build_stg<ND, 1>, build);
    limits_kind<ND, KIND_LJCUT>(force);
    limits_kind<ND, KIND_REPULSION>(force);
    limits_kind<ND, KIND_LJREPULSE>(force);
}

// dynamic shared memory limit of every cell-block kernel, raised once to
// the largest stage (4096 atoms of 16 + 16 bytes); called outside stream
// capture.  A limit is an upper bound only: occupancy follows each launch's
// own size.
int stg_set_smem_limits() {
    const size_t most = 4096 * (sizeof(float4) + sizeof(float4));
    limits_nd<3>(most, most);
    limits_nd<2>(most, most);
    eval_stg_set_smem_limits(most + 4096 * sizeof(uint32_t));   // and the ranks
    return (int)cudaGetLastError();
}

// the tables of every block (after a box change on the same cell grids)
template <int ND>
__global__ void __launch_bounds__(STG_THREADS) k_tables_stg(DevCtx c) {
    __shared__ StgTable T;
    if (blockIdx.x >= c.nblk) return;
    const uint4 bd = c.blk[blockIdx.x];
    stg_setup<ND>(c, c.sys[bd.x], bd, T);
    stg_row_nmax<ND>(c, T);
    stg_store_table(c, T, blockIdx.x);
}

void launch_tables_stg(const DevCtx& c, cudaStream_t s) {
    if (!c.nblk) return;
    if (c.nd == 3) k_tables_stg<3><<<c.nblk, STG_THREADS, 0, s>>>(c);
    else k_tables_stg<2><<<c.nblk, STG_THREADS, 0, s>>>(c);
}

void launch_build_stg(const DevCtx& c, cudaStream_t s) {
    const size_t sm = stg_smem_build(c);
    const unsigned g = c.nblk + c.nsys;
    if (c.nd == 3) {
        if (c.stg_dia) { k_build_stg<3, 1><<<g, STG_THREADS, sm, s>>>(c); }
        else { k_build_stg<3, 0><<<g, STG_THREADS, sm, s>>>(c); }
    } else {
        if (c.stg_dia) { k_build_stg<2, 1><<<g, STG_THREADS, sm, s>>>(c); }
        else { k_build_stg<2, 0><<<g, STG_THREADS, sm, s>>>(c); }
    }
}

constexpr unsigned BAND_CTAS = 2048;

template <int ND, int KIND, int MODE, int PRM>
static void force_stg_split(const DevCtx& c, cudaStream_t s, unsigned g, size_t sm) {
    if (c.stg_lg) launch_after(c, k_force_stg<ND, KIND, MODE, PRM, true>, g, STG_THREADS, sm, s, c);
    else launch_after(c, k_force_stg<ND, KIND, MODE, PRM, false>, g, STG_THREADS, sm, s, c);
}

template <int ND, int KIND, int MODE>
static void force_stg_prm(const DevCtx& c, cudaStream_t s) {
    const size_t sm = stg_smem_force(c);
    const unsigned g = c.nblk + c.nsys;
    switch (c.stg_prm) {
        case 0: force_stg_split<ND, KIND, MODE, 0>(c, s, g, sm); break;
        case 1: force_stg_split<ND, KIND, MODE, 1>(c, s, g, sm); break;
        default: force_stg_split<ND, KIND, MODE, 2>(c, s, g, sm); break;
    }
    if (KIND == KIND_LJCUT) {
        // about one atom in 1500 of an LJ liquid has a pair in the band
        const unsigned bg = std::max(16u, std::min(BAND_CTAS, c.n / 512u));
        switch (c.stg_prm) {
            case 0: launch_after(c, k_band_stg<ND, KIND, MODE, 0>, bg, 32 * BAND_WARPS, 0, s, c); break;
            case 1: launch_after(c, k_band_stg<ND, KIND, MODE, 1>, bg, 32 * BAND_WARPS, 0, s, c); break;
            default: launch_after(c, k_band_stg<ND, KIND, MODE, 2>, bg, 32 * BAND_WARPS, 0, s, c); break;
        }
    }
}

template <int ND, int KIND>
static void force_stg_mode(const DevCtx& c, cudaStream_t s, int mode) {
    if (mode == FM_FORCES_A) force_stg_prm<ND, KIND, FM_FORCES_A>(c, s);
    else force_stg_prm<ND, KIND, FM_FORCES>(c, s);
}

template <int ND>
static void force_stg_kind(const DevCtx& c, cudaStream_t s, int mode) {
    switch (c.kind) {
        case KIND_LJCUT: force_stg_mode<ND, KIND_LJCUT>(c, s, mode); break;
        case KIND_REPULSION: force_stg_mode<ND, KIND_REPULSION>(c, s, mode); break;
        default: force_stg_mode<ND, KIND_LJREPULSE>(c, s, mode); break;
    }
}

void launch_force_stg(const DevCtx& c, cudaStream_t s, int mode) {
    if (c.nd == 3) force_stg_kind<3>(c, s, mode);
    else force_stg_kind<2>(c, s, mode);
}

void launch_expand_stg(const DevCtx& c, cudaStream_t s) {
    if (c.nd == 3) k_expand_stg<3><<<c.nblk, STG_THREADS, 0, s>>>(c);
    else k_expand_stg<2><<<c.nblk, STG_THREADS, 0, s>>>(c);
}

void launch_compress_stg(const DevCtx& c, cudaStream_t s) {
    if (c.nd == 3) k_compress_stg<3><<<c.nblk, STG_THREADS, 0, s>>>(c);
    else k_compress_stg<2><<<c.nblk, STG_THREADS, 0, s>>>(c);
}

}  // namespace parm
