// Interaction quantities (energy, virial, stress, contacts, overlaps, pairs) of
// the mixed path's cell-block lists (staged.cuh).
#include "staged.cuh"

namespace parm {

// ---------------------------------------------------------------------------
// Per-system interaction quantities from the staged lists (EvalWhat, and
// EV_PAIRS: the listed pairs): one CTA per block, the neighbourhood staged as
// for the forces with the atoms' ranks beside it, each pair taken once, for its
// atom of higher rank.  One thread walks a home atom's list and only compares
// ranks: half of the entries belong to the other atom, so the pairs are queued
// per warp and evaluated 32 at a time on full warps (evaluating them in place
// took 143 instructions an entry at 24 active lanes).  A block's pairs belong
// to one system, so the sums need no per-atom place: a block writes its partial
// sums.
// Counts agree with the per-atom kernel's (k_eval32) pair by pair: a pair whose
// energy is near zero or whose distance is near its cut-off, where the last
// bit of the displacement or a quotient may decide, is evaluated with that
// kernel's own arithmetic.
// Measured at 131,072 LJ atoms (one GB300, cold caches): energy 123 us, virial
// 141, stress 238, contacts 89, pairs 51; bound by the staging's latency (no unit
// above half) and, the stress, by its FP64 sums (71 % of the pipe).  (Expanding
// the lists to row-major ones, 101 to 124 us a call, and walking those with a
// thread per atom took 215 us on top on average, 338 for the stress.)
// ---------------------------------------------------------------------------
constexpr uint32_t EVQ = 96;   // queue per warp: fewer than 32 waiting and two entries of each lane

// pair energy of k_eval32 for global atoms i, j (its displacement and law)
template <int ND, int KIND>
__device__ __forceinline__ float eval_exactly(const DevCtx& c, const SysConst& S, uint32_t i, uint32_t j) {
    float4 Ai, Bi, Aj, Bj;
    ld_pos(c.pos, i, Ai, Bi);
    ld_pos(c.pos, j, Aj, Bj);
    const float4 Qi = c.prm32[i], Qj = c.prm32[j];
    float r[3];
    disp3<ND>(S, Ai, Bi, Aj, Bj, r);
    float d2 = r[0] * r[0] + r[1] * r[1];
    if constexpr (ND == 3) d2 += r[2] * r[2];
    const float third = cut_kind<KIND>() ? fmaxf(Qi.z, Qj.z) : 0.5f * (Qi.z + Qj.z);
    const float m6 = cut_kind<KIND>() ? (Qj.z > Qi.z ? Qj.w : Qi.w) : 0.f;
    return energy32<KIND>(d2, Qi.x * Qj.x, 0.5f * (Qi.y + Qj.y), third, m6);
}

// whether a pair's energy e (energy32) is zero or not, or its sign, may hang on
// the last bits of the displacement; NaN counts as in doubt
template <int KIND>
__device__ __forceinline__ bool eval_in_doubt(float e, float d2, float eps, float sig, float third) {
    const float s2 = sig * sig;
    if constexpr (KIND == KIND_REPULSION) {
        return fabsf(d2 - s2) <= 1e-4f * s2 || (d2 <= s2 && !(fabsf(e) > 1e-30f));
    } else {
        const float rsq = d2 / s2, cut2 = KIND == KIND_LJCUT ? third * third : 1.0f;
        return fabsf(rsq - cut2) <= 1e-4f * cut2 || (!(rsq > cut2) && !(fabsf(e) > 1e-4f * eps));
    }
}

// SUMS: energy, virial and stress (FP64 sums); else the counts
template <int ND, int KIND, int PRM, bool SUMS>
__global__ void __launch_bounds__(STG_THREADS, 4) k_eval_stg(DevCtx c, int what) {
    extern __shared__ float4 smem_e[];
    __shared__ StgTable T;
    __shared__ uint32_t queue_s[STG_THREADS / 32][EVQ];   // home atom's local index << 16 | neighbour's
    __shared__ double part[STG_THREADS / 32][9];
    __shared__ uint64_t bar;
    const uint4 bd = c.blk[blockIdx.x];
    const SysConst& S = c.sys[bd.x];
    stg_load_table(c, T, blockIdx.x);
    const int nc = what == EV_STRESS ? ND * ND : 1;
    const bool pairs_only = !SUMS && what == EV_PAIRS;
    // nothing listed in the block (dilute systems)
    uint32_t longest = 0u;
    for (int r = 0; r < T.y1 - T.y0; r++) longest = max(longest, T.hnmax[r]);
    if (longest == 0u) {
        if (threadIdx.x < (uint32_t)nc) c.blk_part[(size_t)blockIdx.x * nc + threadIdx.x] = 0.0;
        return;
    }
    if (!pairs_only) stg_prefetch<ND>(c, T, true);
    const uint32_t cap = c.stg_cap_eval, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    float4* srec = smem_e;
    void* sext = smem_e + cap;
    uint32_t* srank = reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(sext) +
                                                  (size_t)cap * (PRM == 1 ? 4u : (PRM == 2 ? 16u : 0u)));
    // ranks, four pieces' loads in flight per warp
    for (uint32_t p0 = warp; p0 < T.npiece; p0 += 4u * (STG_THREADS / 32)) {
        uint32_t rk[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const uint32_t p = p0 + u * (STG_THREADS / 32);
            rk[u] = p < T.npiece && lane < T.cnt[p] ? __ldg(&c.rank[T.g0[p] + lane]) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; u++) {
            const uint32_t p = p0 + u * (STG_THREADS / 32);
            if (p >= T.npiece) break;
            const uint32_t o = T.off[p];
            if (lane < T.cnt[p] && o + lane < cap) srank[o + lane] = rk[u];
            for (uint32_t t = lane + 32u; t < T.cnt[p] && o + t < cap; t += 32u) srank[o + t] = __ldg(&c.rank[T.g0[p] + t]);
        }
    }
    // (counting the pairs takes the ranks alone; both ways end with a barrier)
    if (pairs_only) __syncthreads();
    else if (!stg_load_bulk<ND, PRM>(c, T, srec, sext, cap, &bar)) return;
    const float* ssig = static_cast<const float*>(sext);
    const float4* sprm = static_cast<const float4*>(sext);
    uint32_t* queue = queue_s[warp];
    // every member has atom 0 of the block's parameters where they are uniform
    const float4 QU = T.nhome ? c.prm32[stg_home<ND, false>(c, T, 0u).i] : make_float4(1.f, 1.f, 1.f, 1.f);
    const float isig2_u = 1.0f / (QU.y * QU.y);
    double acc[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    uint32_t count = 0u, waiting = 0u;
    auto prm = [&](uint32_t q) { return q < cap ? sprm[q] : c.prm32[stg_global(T, q)]; };
    auto sigma = [&](uint32_t q) { return q < cap ? ssig[q] : c.prm32[stg_global(T, q)].y; };
    auto evaluate = [&](uint32_t item) {
        const uint32_t qi = item >> 16, q = item & 0xFFFFu;
        const float4 rec_i = stg_get<ND>(c, S, T, srec, cap, qi), rec_j = stg_get<ND>(c, S, T, srec, cap, q);
        float r[3];
        stg_disp<ND>(stg_wi(rec_i), rec_i, rec_j, r);
        float d2 = fmaf(r[1], r[1], r[0] * r[0]);
        if constexpr (ND == 3) d2 = fmaf(r[2], r[2], d2);
        float eps = QU.x * QU.x, sig = QU.y, isig2 = isig2_u, third = QU.z, m6 = QU.w;
        if constexpr (PRM == 1) {
            sig = 0.5f * (sigma(qi) + sigma(q));
            isig2 = 1.0f / (sig * sig);
        } else if constexpr (PRM == 2) {
            const float4 Qi = prm(qi), Qj = prm(q);
            eps = Qi.x * Qj.x;
            sig = 0.5f * (Qi.y + Qj.y);
            isig2 = 1.0f / (sig * sig);
            third = cut_kind<KIND>() ? fmaxf(Qi.z, Qj.z) : 0.5f * (Qi.z + Qj.z);
            m6 = Qj.z > Qi.z ? Qj.w : Qi.w;
        }
        if (!SUMS || what == EV_ENERGY) {
            float e = energy32<KIND>(d2, eps, sig, third, m6);
            if constexpr (SUMS) {
                acc[0] += f2d_flush(e);
            } else {
                if (eval_in_doubt<KIND>(e, d2, eps, sig, third))
                    e = eval_exactly<ND, KIND>(c, S, stg_global(T, qi), stg_global(T, q));
                count += (what == EV_CONTACTS ? e != 0.0f : e > 0.0f) ? 1u : 0u;
            }
        } else if constexpr (SUMS) {
            bool near_cut;
            const float e12 = (KIND == KIND_REPULSION) ? eps : 12.0f * eps;
            float sc = scale32<KIND>(d2, e12, sig, isig2, third, near_cut);
            if constexpr (cut_kind<KIND>()) {
                if (near_cut) {
                    const float rsq = d2 / (sig * sig);
                    const float ir3 = 1.0f / (rsq * rsq * rsq);
                    sc = lj_beyond_exact_s(c, S, stg_global(T, qi), stg_global(T, q), ND)
                             ? 0.0f : e12 * ir3 * (ir3 - 1.0f) / d2;
                }
            }
            const double rd[3] = {f2d_flush(r[0]), f2d_flush(r[1]), f2d_flush(r[2])};
            const double f[3] = {f2d_flush(r[0] * sc), f2d_flush(r[1] * sc), f2d_flush(r[2] * sc)};
            // products of two FP32 values are exact in FP64
            if (what == EV_VIRIAL) {
                double p = __fma_rn(rd[1], f[1], rd[0] * f[0]);
                if constexpr (ND == 3) p = __fma_rn(rd[2], f[2], p);
                acc[0] += p;
            } else {
#pragma unroll
                for (int a = 0; a < ND; a++)
#pragma unroll
                    for (int b = 0; b < ND; b++) acc[a * ND + b] = __fma_rn(rd[a], f[b], acc[a * ND + b]);
            }
        }
    };
    for (uint32_t h0 = threadIdx.x - lane; h0 < T.nhome; h0 += STG_THREADS) {   // uniform in the warp
        HomeAtom a{};
        uint32_t nn = 0u, ri = 0u;
        if (h0 + lane < T.nhome) {
            a = stg_home<ND, false>(c, T, h0 + lane);
            nn = c.nnb[a.i];
            ri = c.rank[a.i];
        }
        // the pair is this atom's: the neighbour's rank is lower
        auto of_mine = [&](uint32_t q) {
            if (q >= T.total) {   // inconsistent list (never): reported, skipped
                stg_check(c, T, q, a.qi);
                return false;
            }
            return (q < cap ? srank[q] : c.rank[stg_global(T, q)]) < ri;
        };
        // the list's 32-bit words of two entries, each loaded two words ahead
        const uint32_t nmax = __reduce_max_sync(0xFFFFFFFFu, nn), nw = (nn + 1u) >> 1;
        const uint32_t* row = reinterpret_cast<const uint32_t*>(c.nbr16) + ((size_t)a.s0 * c.maxnb >> 1) + a.hs;
        uint32_t w0 = nw > 0u ? __ldg(row) : 0u, w1 = nw > 1u ? __ldg(row + a.H) : 0u;
#pragma unroll 1
        for (uint32_t p = 0; 2u * p < nmax; p++) {
            const uint32_t word = w0;
            w0 = w1;
            w1 = p + 2u < nw ? __ldg(row + (size_t)(p + 2u) * a.H) : 0u;
            const bool v0 = 2u * p < nn, v1 = 2u * p + 1u < nn;
            if (pairs_only) {
                count += (v0 && of_mine(word & 0xFFFFu) ? 1u : 0u) + (v1 && of_mine(word >> 16) ? 1u : 0u);
                continue;
            }
            const bool m0 = v0 && of_mine(word & 0xFFFFu), m1 = v1 && of_mine(word >> 16);
            const uint32_t k0 = __ballot_sync(0xFFFFFFFFu, m0), k1 = __ballot_sync(0xFFFFFFFFu, m1);
            const uint32_t below = (1u << lane) - 1u;
            if (m0) queue[waiting + __popc(k0 & below)] = (a.qi << 16) | (word & 0xFFFFu);
            waiting += __popc(k0);
            if (m1) queue[waiting + __popc(k1 & below)] = (a.qi << 16) | (word >> 16);
            waiting += __popc(k1);
            __syncwarp();
            while (waiting >= 32u) {
                waiting -= 32u;
                evaluate(queue[waiting + lane]);
                __syncwarp();
            }
        }
    }
    if (!pairs_only) {
        __syncwarp();
        if (lane < waiting) evaluate(queue[lane]);
    }
    if constexpr (!SUMS) acc[0] = (double)count;
    // fixed-order sums over the block
#pragma unroll
    for (int q = 0; q < (SUMS ? ND * ND : 1); q++) {
        if (q < nc) {
            double v = acc[q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
            if (lane == 0) part[warp][q] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)nc) {
        double v = part[0][threadIdx.x];
        for (uint32_t w = 1; w < STG_THREADS / 32; w++) v += part[w][threadIdx.x];
        c.blk_part[(size_t)blockIdx.x * nc + threadIdx.x] = v;
    }
}

static size_t stg_smem_eval(const DevCtx& c) {
    const size_t ext = c.stg_prm == 1 ? sizeof(float) : (c.stg_prm == 2 ? sizeof(float4) : 0);
    return (size_t)c.stg_cap_eval * (sizeof(float4) + ext + sizeof(uint32_t));
}

template <int ND, int KIND, int PRM>
static void limits_prm(int sm) {
    cudaFuncSetAttribute(k_eval_stg<ND, KIND, PRM, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    cudaFuncSetAttribute(k_eval_stg<ND, KIND, PRM, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
}
template <int ND, int KIND>
static void limits_kind(int sm) {
    limits_prm<ND, KIND, 0>(sm);
    limits_prm<ND, KIND, 1>(sm);
    limits_prm<ND, KIND, 2>(sm);
}
template <int ND>
static void limits_nd(int sm) {
    limits_kind<ND, KIND_LJCUT>(sm);
    limits_kind<ND, KIND_REPULSION>(sm);
    limits_kind<ND, KIND_LJREPULSE>(sm);
}
void eval_stg_set_smem_limits(size_t most) {
    limits_nd<3>((int)most);
    limits_nd<2>((int)most);
}

template <int ND, int KIND, int PRM>
static void eval_stg_prm(const DevCtx& c, cudaStream_t s, int what) {
    const size_t sm = stg_smem_eval(c);
    if (what == EV_ENERGY || what == EV_VIRIAL || what == EV_STRESS)
        k_eval_stg<ND, KIND, PRM, true><<<c.nblk, STG_THREADS, sm, s>>>(c, what);
    else
        k_eval_stg<ND, KIND, PRM, false><<<c.nblk, STG_THREADS, sm, s>>>(c, what);
}
template <int ND, int KIND>
static void eval_stg_kind(const DevCtx& c, cudaStream_t s, int what) {
    switch (c.stg_prm) {
        case 0: eval_stg_prm<ND, KIND, 0>(c, s, what); break;
        case 1: eval_stg_prm<ND, KIND, 1>(c, s, what); break;
        default: eval_stg_prm<ND, KIND, 2>(c, s, what); break;
    }
}
template <int ND>
static void eval_stg_nd(const DevCtx& c, cudaStream_t s, int what) {
    if (c.kind == KIND_LJCUT) eval_stg_kind<ND, KIND_LJCUT>(c, s, what);
    else if (c.kind == KIND_REPULSION) eval_stg_kind<ND, KIND_REPULSION>(c, s, what);
    else eval_stg_kind<ND, KIND_LJREPULSE>(c, s, what);
}

void launch_eval_stg(const DevCtx& c, cudaStream_t s, int what) {
    if (c.nd == 3) eval_stg_nd<3>(c, s, what);
    else eval_stg_nd<2>(c, s, what);
}

}  // namespace parm
