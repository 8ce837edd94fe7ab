// Neighbour-list maintenance on the GPU.
//
// Reference behaviour being reproduced (wackywendell/parm):
//   NeighborList::update_list (src/trackers.cpp:19-85): a rebuild is needed
//   when the two largest displacements since the last build sum to >= skin;
//   a rebuild keeps every pair with |diff(x_i, x_j)| < (d_i + d_j)/2 + skin
//   (strict <, minimum image per OriginBox::diff, src/box.hpp:103) and not
//   excluded by NeighborList::ignore (src/trackers.hpp:190-193).
// The reference tests all N(N-1)/2 pairs.  Here a rebuild is a counting sort
// of the atoms by cell (cells no narrower than the largest list radius),
// followed by a scan of the 3^d neighbouring cells per atom.  Candidate
// distances are screened in FP32; only candidates within 2e-4 (relative) of
// the threshold are decided with the exact FP64 test, so the pair set is
// identical to the reference's.
//
// Compiled with -fmad=false: every FP64 expression here must round exactly
// like the reference's unfused CPU arithmetic.
#include <algorithm>

#include "parm_check.cuh"

namespace parm {

template <int ND>
__device__ __forceinline__ typename DVec<ND>::T ldx(const void* p, uint32_t i) {
    return static_cast<const typename DVec<ND>::T*>(p)[i];
}

__device__ __forceinline__ void posq_split(double x, float& X, float& xf) {
    double t = trunc(x * 8.0) * 0.125;   // exact: scaling by powers of two, truncation
    X = (float)t;                         // exact while |x| < 2^21
    xf = (float)(x - t);                  // x - t is exact; one rounding to FP32
}

// ---------------------------------------------------------------------------
// arm: decide, per system, whether this step starts with a rebuild
// ---------------------------------------------------------------------------
__global__ void k_arm(DevCtx c, int count_step, int use_cond, cudaGraphConditionalHandle handle) {
    arm_systems(c, blockDim.x, count_step, use_cond, handle);
}

// ---------------------------------------------------------------------------
// rebuild chain (every kernel skips systems whose flag is clear)
// ---------------------------------------------------------------------------
template <int ND>
__global__ void k_bin(DevCtx c) {
    // every lane of the warp reaches the cell-count update below (the grid is
    // whole warps), so the lanes that bin a member can be counted by a ballot
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t s = i < c.n ? c.atom_sys[i] : 0u;
    const bool live = i < c.n && c.flag[s];
    const bool member = live && c.rank[i] != NOT_MEMBER;
    uint32_t b = 0u, slot = 0u;
    if (live && !member) {
        b = c.bucket_off[s] + c.sys[s].ncell;
        slot = c.nm_rank[c.orig[i]];
    }
    if (member) {
        const SysConst& S = c.sys[s];
        typename DVec<ND>::T xi = ldx<ND>(c.x, i);
        double xs[3] = {xi.x, xi.y, 0.0};
        if constexpr (ND == 3) xs[2] = reinterpret_cast<const double*>(&xi)[2];
        int ci[3] = {0, 0, 0};
        bool bad = false;
#pragma unroll
        for (int d = 0; d < ND; d++) {
            double t = xs[d] * S.invL[d];
            if (!isfinite(t)) { bad = true; t = 0.0; }
            double fr = t - floor(t);              // wrapped fraction in [0, 1]
            int cc = (int)(fr * (double)S.nc[d]);
            cc = cc < 0 ? 0 : (cc >= S.nc[d] ? S.nc[d] - 1 : cc);
            ci[d] = cc;
        }
        if (bad) atomicOr(c.status, ST_NONFINITE);
        b = c.bucket_off[s] + cell_row(S, ci[1], ci[2]) * (uint32_t)S.nc[0] + (uint32_t)ci[0];
    }
    // one atomic per distinct cell of the warp (atoms arrive in cell order,
    // so a warp holds two or three cells): the lanes of a cell take
    // consecutive slots from its count
    const uint32_t mem = __ballot_sync(0xFFFFFFFFu, member);
    if (member) {
        const uint32_t lane = threadIdx.x & 31u;
        const uint32_t peers = __match_any_sync(mem, b);
        const uint32_t leader = (uint32_t)__ffs(peers) - 1u;
        uint32_t first = 0u;
        if (lane == leader) first = atomicAdd(&c.cell_count[b], (uint32_t)__popc(peers));
        first = __shfl_sync(peers, first, leader);
        slot = first + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    }
    if (live) {
        c.bucket[i] = b;
        c.cslot[i] = slot;
    }
}

// ---------------------------------------------------------------------------
// Cell offsets: a segmented exclusive scan of the bucket counts over all
// buckets, one segment per system (its first bucket starts a segment), in
// two passes (block aggregates; offsets, where each block first sums the
// aggregates before its own: a pass for that sum in between cost 20,011 disks,
// which rebuild every other step, 0.8 us of their 49 us a step).  Only buckets of
// flagged systems are written, and their counts cleared; other systems have none.
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_CHUNK = SCAN_THREADS * SCAN_ITEMS;
constexpr uint32_t SCAN_ONE = 1;   // chunks up to which one block scans them all (three: 6 us slower than the passes)

struct SegPair {
    uint32_t f;  // segment starts in this span
    uint32_t v;  // sum since the last segment start
};

__device__ __forceinline__ SegPair seg_combine(SegPair a, SegPair b) {
    return {a.f | b.f, b.f ? b.v : a.v + b.v};
}

// block-wide inclusive scan of one pair per thread; returns the exclusive
// carry for this thread and the block aggregate
__device__ __forceinline__ SegPair seg_block_scan(SegPair x, SegPair& aggregate) {
    __shared__ SegPair wsum[SCAN_THREADS / 32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    SegPair inc = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        SegPair o;
        o.f = __shfl_up_sync(0xFFFFFFFFu, inc.f, off);
        o.v = __shfl_up_sync(0xFFFFFFFFu, inc.v, off);
        if (lane >= (unsigned)off) inc = seg_combine(o, inc);
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        SegPair w = lane < SCAN_THREADS / 32 ? wsum[lane] : SegPair{0u, 0u};
        SegPair wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            SegPair o;
            o.f = __shfl_up_sync(0xFFFFFFFFu, wi.f, off);
            o.v = __shfl_up_sync(0xFFFFFFFFu, wi.v, off);
            if (lane >= (unsigned)off) wi = seg_combine(o, wi);
        }
        if (lane < SCAN_THREADS / 32) wsum[lane] = wi;   // inclusive over warps
    }
    __syncthreads();
    aggregate = wsum[SCAN_THREADS / 32 - 1];
    // exclusive carry = (inclusive of previous warps) + (inclusive of earlier lanes)
    SegPair prev_w = warp > 0 ? wsum[warp - 1] : SegPair{0u, 0u};
    SegPair prev_l;
    prev_l.f = __shfl_up_sync(0xFFFFFFFFu, inc.f, 1);
    prev_l.v = __shfl_up_sync(0xFFFFFFFFu, inc.v, 1);
    if (lane == 0) prev_l = SegPair{0u, 0u};
    SegPair carry = seg_combine(prev_w, prev_l);
    __syncthreads();
    return carry;
}

// offset of bucket b from the segmented prefix `run` before its item
__device__ __forceinline__ void bucket_offset(const DevCtx& c, uint32_t b, const SegPair& item, const SegPair& run) {
    const uint32_t s = c.bucket_sys[b];
    if (!c.flag[s]) return;
    c.cell_start[b] = c.sys[s].atom_off + (item.f ? 0u : run.v);   // exclusive, restarted per system
    c.cell_count[b] = 0u;
    if (item.f && c.half_cnt) c.half_cnt[s] = 0u;   // the rebuild hands out the system's pair slots anew
}

__device__ __forceinline__ SegPair bucket_item(const DevCtx& c, uint32_t b) {
    if (b >= c.nbucket) return {0u, 0u};
    const uint32_t s = c.bucket_sys[b];
    return {b == c.bucket_off[s] ? 1u : 0u, c.cell_count[b]};
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_blocks(DevCtx c) {
    const uint32_t base = blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    SegPair t{0u, 0u};
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) t = seg_combine(t, bucket_item(c, base + k));
    SegPair agg;
    seg_block_scan(t, agg);
    if (threadIdx.x == 0) {
        c.scan_aux[2 * blockIdx.x] = agg.f;
        c.scan_aux[2 * blockIdx.x + 1] = agg.v;
    }
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_write(DevCtx c) {
    const uint32_t base = blockIdx.x * SCAN_CHUNK + threadIdx.x * SCAN_ITEMS;
    SegPair items[SCAN_ITEMS];
    SegPair t{0u, 0u};
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        items[k] = bucket_item(c, base + k);
        t = seg_combine(t, items[k]);
    }
    SegPair agg, before{0u, 0u};
    for (uint32_t b0 = 0; b0 < blockIdx.x; b0 += SCAN_THREADS) {
        const uint32_t b = b0 + threadIdx.x;
        const bool on = b < blockIdx.x;
        seg_block_scan(on ? SegPair{c.scan_aux[2 * b], c.scan_aux[2 * b + 1]} : SegPair{0u, 0u}, agg);
        before = seg_combine(before, agg);
    }
    SegPair run = seg_combine(before, seg_block_scan(t, agg));
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        const uint32_t b = base + k;
        if (b >= c.nbucket) break;
        bucket_offset(c, b, items[k], run);
        run = seg_combine(run, items[k]);
    }
}

// the whole scan in one block
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_one(DevCtx c) {
    SegPair carry{0u, 0u};
    for (uint32_t b0 = 0; b0 < c.nbucket; b0 += SCAN_CHUNK) {
        const uint32_t base = b0 + threadIdx.x * SCAN_ITEMS;
        SegPair items[SCAN_ITEMS];
        SegPair t{0u, 0u};
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            items[k] = bucket_item(c, base + k);
            t = seg_combine(t, items[k]);
        }
        SegPair agg;
        SegPair run = seg_combine(carry, seg_block_scan(t, agg));
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            if (base + k >= c.nbucket) break;
            bucket_offset(c, base + k, items[k], run);
            run = seg_combine(run, items[k]);
        }
        carry = seg_combine(carry, agg);
    }
}

// the entries of atom o of the old order, at place k of the new one in bucket b
template <int ND>
__device__ __forceinline__ void move_atom(const DevCtx& c, uint32_t o, uint32_t k, uint32_t rk, uint32_t b) {
    using V = typename DVec<ND>::T;
    static_cast<V*>(c.x2)[k] = static_cast<const V*>(c.x)[o];
    static_cast<V*>(c.v2)[k] = static_cast<const V*>(c.v)[o];
    static_cast<V*>(c.a2)[k] = static_cast<const V*>(c.a)[o];
    if (c.prec != PREC_MIXED) static_cast<V*>(c.f2)[k] = static_cast<const V*>(c.f)[o];   // FP64 forces: FP64 path only
    c.f32b[k] = c.f32[o];
    // arrays whose entries are all equal are left as they are (copy back too)
    if (*c.m_mixed) {
        c.m2[k] = c.m[o];
        c.invm32b[k] = c.invm32[o];
    }
    if (!c.same_prm) {
        c.prm2[k] = c.prm[o];
        c.prm32b[k] = c.prm32[o];
        c.diam2[k] = c.diam[o];
    }
    c.rank2[k] = rk;
    c.orig2[k] = c.orig[o];
    c.bucket2[k] = b;
}

// Members into their cells, in any order; non-members, whose order nm_rank
// gives, with all their entries to their place at the system's end, a thread
// each (rebuild with 399,000 of 400,000 atoms outside the list: 0.91 ms; with a
// warp for all of them 55.9 ms).
template <int ND>
__global__ void k_scatter(DevCtx c) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    uint32_t s = c.atom_sys[i];
    if (!c.flag[s]) return;
    const uint32_t b = c.bucket[i], k = c.cell_start[b] + c.cslot[i];
    if (b - c.bucket_off[s] == c.sys[s].ncell) move_atom<ND>(c, i, k, NOT_MEMBER, b);
    else c.perm[k] = i;
}

// Permutation of the members' arrays into their new order: the order inside a
// cell is ascending neighbour-list rank, so each of LANES lanes holds one of
// the cell's scattered atoms, counts the atoms of the cell ranked before it,
// LANES at a time, and moves its atom's entries to that place.  Bound by those
// moves' memory latency, so few lanes may idle: with a warp per cell / eight /
// four lanes, 400,000 disks in cells of one 219 / 74 / 45 us, of two 124 / 40 /
// 35 us, 48 WCA replicas (427,107 atoms, two a cell) 98 / 34 / 25 us, 65,536
// disks 26.8 / 10.9 / 13.5 us, 20,011 disks 14.7 / 9.4 / 11.9 us; 343,000 LJ
// atoms (17 a cell) 18.9 / 26.2 / 44.1 us; 48 packings of 64 to 4096 spheres,
// one cell of 86 among 10,693: a warp / sixteen / eight lanes 25.2 / 21.4 / 32.0
// us.  `parts` groups share a cell, each taking every parts-th
// LANES of its atoms: one for cells of up to 32 atoms, more where few-cell boxes
// put hundreds in one (rebuild of 1000 / 3000 atoms in one cell: 0.31 / 2.0 ms;
// with one warp for it 0.83 / 6.5 ms).  (Sort and move as two kernels cost a
// batch of 48 replicas, one of which rebuilds nearly every step, 1 % of the
// step.)
template <int ND, uint32_t LANES>
__global__ void k_sortgather(DevCtx c, uint32_t parts) {
    const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) / LANES, lane = threadIdx.x % LANES;
    const uint32_t b = parts == 1u ? w : w / parts, part = w - b * parts;
    uint32_t lo = 0u, cnt = 0u;
    if (b < c.nbucket) {
        const uint32_t s = c.bucket_sys[b];
        // (not: non-members, buckets past a grid that has shrunk)
        if (c.flag[s] && b - c.bucket_off[s] < c.sys[s].ncell) {
            lo = c.cell_start[b];
            cnt = c.cell_start[b + 1] - lo;
        }
    }
    const uint32_t most = LANES == 32u ? cnt : __reduce_max_sync(0xFFFFFFFFu, cnt);   // uniform in the warp
    // (the groups of a warp may be different parts of a cell: all stay for the shuffles of the longest)
    for (uint32_t q0 = LANES * part; LANES == 32u ? q0 < most : __any_sync(0xFFFFFFFFu, q0 < most) != 0;
         q0 += LANES * parts) {
        const bool on = q0 + lane < cnt;
        const uint32_t o = on ? c.perm[lo + q0 + lane] : 0u;
        const uint32_t rk = on ? c.rank[o] : 0xFFFFFFFFu;
        uint32_t pos = 0u;
        for (uint32_t t0 = 0; t0 < most; t0 += 4u * LANES) {
            uint32_t kt[4];   // four groups of ranks, their loads in flight together
#pragma unroll
            for (uint32_t g = 0; g < 4u; g++) {
                const uint32_t t = t0 + g * LANES;
                kt[g] = rk;
                if (t != q0) kt[g] = t + lane < cnt ? c.rank[c.perm[lo + t + lane]] : 0xFFFFFFFFu;
            }
#pragma unroll
            for (uint32_t g = 0; g < 4u; g++) {
                const uint32_t t = t0 + g * LANES;
                if (t >= most) break;   // uniform in the warp
                const uint32_t m = min(LANES, most - t);
                for (uint32_t j = 0; j < m; j++) pos += __shfl_sync(0xFFFFFFFFu, kt[g], j, LANES) < rk ? 1u : 0u;
            }
        }
        if (on) move_atom<ND>(c, o, lo + pos, rk, b);
    }
}

// STAGED: c.staged (apart: the one that forms the records of the cell blocks
// then carries none of the other's FP64 operations, which the compiler had
// executed for both: 45.6 -> 26.3 us at 343,000 LJ atoms)
template <int ND, bool STAGED>
__global__ void k_copyback(DevCtx c) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    uint32_t s = c.atom_sys[k];
    if (!c.flag[s]) return;
    using V = typename DVec<ND>::T;
    V xk = static_cast<const V*>(c.x2)[k];
    static_cast<V*>(c.x)[k] = xk;
    static_cast<V*>(c.lastloc)[k] = xk;
    static_cast<V*>(c.v)[k] = static_cast<const V*>(c.v2)[k];
    static_cast<V*>(c.a)[k] = static_cast<const V*>(c.a2)[k];
    if (c.prec != PREC_MIXED) static_cast<V*>(c.f)[k] = static_cast<const V*>(c.f2)[k];
    c.f32[k] = c.f32b[k];
    if (*c.m_mixed) {
        c.m[k] = c.m2[k];
        c.invm32[k] = c.invm32b[k];
    }
    double dk;
    if (!c.same_prm) {
        c.prm[k] = c.prm2[k];
        c.prm32[k] = c.prm32b[k];
        dk = c.diam2[k];
        c.diam[k] = dk;
    } else {
        dk = c.diam[k];   // every atom's
    }
    c.rank[k] = c.rank2[k];
    uint32_t og = c.orig2[k];
    c.orig[k] = og;
    c.slot[og] = k;
    c.bucket[k] = c.bucket2[k];
    const double* xs = reinterpret_cast<const double*>(&xk);
    float4 A, B;
    posq_split(xs[0], A.x, B.x);
    posq_split(xs[1], A.y, B.y);
    if constexpr (ND == 3) posq_split(xs[2], A.z, B.z); else { A.z = 0.f; B.z = 0.f; }
    A.w = (float)dk;
    B.w = 0.f;
    c.pos[2 * (size_t)(k)] = A;
    c.pos[2 * (size_t)(k) + 1] = B;
    if constexpr (STAGED) {
        // cell-block record in the frame of this build
        float4 fr = make_float4(0.f, 0.f, 0.f, __uint_as_float(REC_BIAS | (REC_BIAS << 12) | (REC_BIAS << 22)));
        if (c.rank[k] != NOT_MEMBER) {
            const SysConst& S = c.sys[s];
            uint32_t ci[3];
            cell_coords(S, c.bucket[k] - c.bucket_off[s], ci);
            bool ok;
            fr = rec_frame<ND>(S, ci, A, B, ok);
            if (!ok) atomicOr(c.status, ST_IMAGE_RANGE);
        }
        c.rframe[k] = fr;
        c.rec[k] = make_record(A, B, fr);
    }
    // position relative to the lower corner of its cell, for the warp list
    // build (the cell-block build stages its own positions)
    if (!STAGED && c.rank[k] != NOT_MEMBER) {
        const SysConst& S = c.sys[s];
        const uint32_t myb = c.bucket[k] - c.bucket_off[s];
        uint32_t ci[3];
        cell_coords(S, myb, ci);
        float pr[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int d = 0; d < ND; d++) {
            double t = xs[d] * S.invL[d];
            double fr = t - floor(t);
            pr[d] = (float)(fr * S.L[d] - (double)ci[d] * S.cellw[d]);
        }
        c.posw[k] = make_float4(pr[0], pr[1], pr[2], (float)dk);
    }
}

__device__ __forceinline__ bool is_excluded(const DevCtx& c, uint32_t oi, uint32_t oj) {
    if (!c.excl_off) return false;
    for (uint32_t e = c.excl_off[oi]; e < c.excl_off[oi + 1]; e++)
        if (c.excl_list[e] == oj) return true;
    return false;
}

// exact reference test: diff(x_i, x_j).norm() < (d_i + d_j)/2 + skin
template <int ND>
__device__ __noinline__ bool keep_exact(const DevCtx& c, const SysConst& S, uint32_t i, uint32_t j) {
    typename DVec<ND>::T xi = ldx<ND>(c.x, i), xj = ldx<ND>(c.x, j);
    const double* a = reinterpret_cast<const double*>(&xi);
    const double* bb = reinterpret_cast<const double*>(&xj);
    double r[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < ND; d++) r[d] = remainder_exact(a[d] - bb[d], S.L[d], S.invL[d], S.halfL[d]);
    double sq = r[0] * r[0] + r[1] * r[1];
    if constexpr (ND == 3) sq = sq + r[2] * r[2];
    double diam = (c.diam[i] + c.diam[j]) / 2;
    return sqrt(sq) < (diam + S.skin);
}

// Full neighbour lists of a flagged system's member atoms (row-major:
// nbr[i * maxnb + k]), one warp per cell with warp-ballot compaction.
// The candidates of the 3^d stencil cells are numbered consecutively (stencil
// order, then cell order); the warp takes 32 candidates at a time, one per
// lane, and tests all of them against each home atom in turn.  The accepted
// candidates of a home atom are appended in candidate order by a ballot and a
// population count, so the lists are deterministic and written coalesced.
// Positions are relative to each cell's lower corner: a candidate in the
// stencil cell at offset (dx,dy,dz) is displaced by (dx,dy,dz) * cell width in
// the periodic continuation of the grid (axes with a single cell take a
// per-pair minimum image instead).  Distances are screened in FP32; candidates
// within 2e-4 (relative) of the threshold get the exact FP64 reference test.
// `parts` warps share a cell, each taking every parts-th group of `per` of its
// home atoms (grids of a few cells with tens of atoms each would otherwise run
// on a few warps: 296 -> 25 us at 1000 LJ atoms in 27 cells).
constexpr int BUILD_WARPS = 4;
template <int ND, bool WRAP>
__global__ void __launch_bounds__(BUILD_WARPS * 32) k_build(DevCtx c, uint32_t parts, uint32_t per) {
    __shared__ float4 home[BUILD_WARPS][32];
    __shared__ uint32_t pre[BUILD_WARPS][32];
    __shared__ uint32_t jst[BUILD_WARPS][32];
    __shared__ float4 soff[BUILD_WARPS][32];
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint32_t wid = blockIdx.x * BUILD_WARPS + wib;
    const uint32_t b = wid / parts, part = wid % parts;   // bucket, share of its home atoms
    if (b >= c.nbucket) return;
    const uint32_t s = c.bucket_sys[b];
    if (!c.flag[s]) return;
    const SysConst& S = c.sys[s];
    const uint32_t b0 = c.bucket_off[s];
    const uint32_t myb = b - b0;
    if (myb >= S.ncell) {
        // non-member bucket: these atoms have no neighbours
        for (uint32_t i = c.cell_start[b] + lane; i < S.atom_off + S.natoms; i += 32) c.nnb[i] = 0u;
        return;
    }
    const uint32_t cs = c.cell_start[b], ce = c.cell_start[b + 1];
    if (cs + part * per >= ce) return;
    const int nc0 = S.nc[0], nc1 = S.nc[1], nc2 = S.nc[2];
    uint32_t ci[3];
    cell_coords(S, myb, ci);
    const int ci0 = (int)ci[0], ci1 = (int)ci[1], ci2 = (int)ci[2];
    const int r0 = nc0 >= 3 ? 1 : 0, r1 = nc1 >= 3 ? 1 : 0;
    const int r2 = (ND == 3 && nc2 >= 3) ? 1 : 0;
    const int w0 = 2 * r0 + 1, w1 = 2 * r1 + 1, w2 = 2 * r2 + 1;
    const uint32_t nst = (uint32_t)(w0 * w1 * w2);
    // stencil table: lane t describes stencil cell t
    uint32_t cntl = 0;
    if (lane < nst) {
        const int dx = (int)(lane % (uint32_t)w0) - r0;
        const int dy = (int)((lane / (uint32_t)w0) % (uint32_t)w1) - r1;
        const int dz = (int)(lane / (uint32_t)(w0 * w1)) - r2;
        int cx = ci0 + dx, cy = ci1 + dy, cz = ci2 + dz;
        cx = cx < 0 ? cx + nc0 : (cx >= nc0 ? cx - nc0 : cx);
        cy = cy < 0 ? cy + nc1 : (cy >= nc1 ? cy - nc1 : cy);
        cz = cz < 0 ? cz + nc2 : (cz >= nc2 ? cz - nc2 : cz);
        const uint32_t cb = b0 + cell_row(S, cy, cz) * (uint32_t)nc0 + (uint32_t)cx;
        const uint32_t js = c.cell_start[cb];
        cntl = c.cell_start[cb + 1] - js;
        jst[wib][lane] = js;
        soff[wib][lane] = make_float4((float)dx * S.cellw32[0], (float)dy * S.cellw32[1],
                                      (float)dz * S.cellw32[2], 0.f);
    }
    uint32_t incl = cntl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    pre[wib][lane] = incl - cntl;
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    __syncwarp();

    // per-pair minimum image only along axes with a single cell (WRAP kernels)
    const bool wrap0 = WRAP && r0 == 0, wrap1 = WRAP && r1 == 0, wrap2 = WRAP && (ND == 3) && r2 == 0;
    const float kShift = 12582912.0f;
    const float skin32 = (float)S.skin;
    const bool uni_thr = c.uniform & UNI_DIAM;
    const uint32_t maxnb = c.maxnb;
    for (uint32_t hb = cs + part * per; hb < ce; hb += parts * per) {
        const uint32_t mh = min(per, ce - hb);
        if (lane < mh) home[wib][lane] = c.posw[hb + lane];
        uint32_t mycnt = 0;   // neighbours found so far for home atom hb + lane
        __syncwarp();
        const float4 H0 = home[wib][0];
        const float t2u = (H0.w + skin32) * (H0.w + skin32);
        for (uint32_t base = 0; base < total; base += 32) {
            const uint32_t q = base + lane;
            const bool valid = q < total;
            uint32_t j = 0xFFFFFFFFu;
            float4 Q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (valid) {
                // the last stencil cell that starts at or before q (unused lanes
                // hold the total)
                uint32_t st = 0;
#pragma unroll
                for (uint32_t h = 16; h; h >>= 1)
                    if (pre[wib][st + h] <= q) st += h;
                j = jst[wib][st] + (q - pre[wib][st]);
                const float4 R = c.posw[j];
                const float4 O = soff[wib][st];
                Q = make_float4(R.x + O.x, R.y + O.y, R.z + O.z, R.w);
            }
            for (uint32_t h = 0; h < mh; h++) {
                const float4 P = home[wib][h];
                float d0 = P.x - Q.x, d1 = P.y - Q.y, d2c = 0.f;
                if (wrap0) d0 = __fmaf_rn(-__fsub_rn(__fmaf_rn(d0, S.invLf[0], kShift), kShift), S.Lhi[0], d0);
                if (wrap1) d1 = __fmaf_rn(-__fsub_rn(__fmaf_rn(d1, S.invLf[1], kShift), kShift), S.Lhi[1], d1);
                if constexpr (ND == 3) {
                    d2c = P.z - Q.z;
                    if (wrap2) d2c = __fmaf_rn(-__fsub_rn(__fmaf_rn(d2c, S.invLf[2], kShift), kShift), S.Lhi[2], d2c);
                }
                const float rr = d0 * d0 + d1 * d1 + d2c * d2c;
                float t2 = t2u;
                if (!uni_thr) {
                    const float thr = 0.5f * (P.w + Q.w) + skin32;
                    t2 = thr * thr;
                }
                const uint32_t i = hb + h;
                bool keep = valid && rr < t2 * 0.9998f && j != i;
                const bool band = valid && !keep && rr <= t2 * 1.0002f && j != i;
                if (__any_sync(0xFFFFFFFFu, band)) {   // rare: exact reference test
                    if (band) keep = keep_exact<ND>(c, S, i, j);
                }
                if (c.excl_off) {
                    if (keep && is_excluded(c, c.orig[i], c.orig[j])) keep = false;
                }
                const uint32_t mask = __ballot_sync(0xFFFFFFFFu, keep);
                if (mask) {
                    const uint32_t ch = __shfl_sync(0xFFFFFFFFu, mycnt, h);
                    if (keep) {
                        const uint32_t pos = ch + __popc(mask & ((1u << lane) - 1u));
                        if (pos < maxnb) c.nbr[(size_t)i * maxnb + pos] = j;
                    }
                    if (lane == h) mycnt += __popc(mask);
                }
            }
        }
        if (lane < mh) {
            if (mycnt > maxnb) {
                atomicOr(c.status, ST_NBR_OVERFLOW);
                mycnt = maxnb;
            }
            c.nnb[hb + lane] = mycnt;
        }
        __syncwarp();
    }
}

// All-pairs list build of the handles with a LeesEdwardsBox (FP64 path): the
// sheared images do not follow the cell stencil, so every member atom tests
// every member of its system with the reference's own test (trackers.cpp:
// 59-69: diff(x_i, x_j).norm() < (d_i + d_j)/2 + skin), as the reference's
// O(N^2) list build does; k_sort_lists then orders each list by rank.
template <int ND>
__global__ void k_build_lees(DevCtx c) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const uint32_t s = c.atom_sys[i];
    if (!c.flag[s]) return;
    if (c.rank[i] == NOT_MEMBER) {
        c.nnb[i] = 0u;
        return;
    }
    const SysConst& S = c.sys[s];
    typename DVec<ND>::T xv = ldx<ND>(c.x, i);
    const double* xi = reinterpret_cast<const double*>(&xv);
    const double di = c.diam[i];
    const uint32_t maxnb = c.maxnb;
    uint32_t cnt = 0;
    for (uint32_t j = S.atom_off; j < S.atom_off + S.natoms; j++) {
        if (j == i || c.rank[j] == NOT_MEMBER) continue;
        typename DVec<ND>::T yv = ldx<ND>(c.x, j);
        const double* xj = reinterpret_cast<const double*>(&yv);
        double r[3] = {0.0, 0.0, 0.0};
        if (S.lees) {
            lees_diff<ND>(S, xi, xj, r);
        } else {
#pragma unroll
            for (int d = 0; d < ND; d++) r[d] = remainder_exact(xi[d] - xj[d], S.L[d], S.invL[d], S.halfL[d]);
        }
        double sq = r[0] * r[0] + r[1] * r[1];
        if constexpr (ND == 3) sq = sq + r[2] * r[2];
        const double diam = (di + c.diam[j]) / 2;
        if (!(sqrt(sq) < (diam + S.skin))) continue;
        if (c.excl_off && is_excluded(c, c.orig[i], c.orig[j])) continue;
        if (cnt < maxnb) c.nbr[(size_t)i * maxnb + cnt] = j;
        cnt++;
    }
    if (cnt > maxnb) {
        atomicOr(c.status, ST_NBR_OVERFLOW);
        cnt = maxnb;
    }
    c.nnb[i] = cnt;
}

// ---------------------------------------------------------------------------
// Shared-memory tiles for the mixed-precision pair kernel (built after the
// lists).  A tile is TILE_ATOMS consecutive atoms of one system.  Its frame
// origin is the coarse position A0 of its first atom; atom i sits in the frame
// at X_i - m_i L (m_i rounds (X_i - A0)/L), and its neighbour j, whose pair
// image is n_ij = round((X_i - X_j)/L), at X_j + (n_ij - m_i) L.  The tile's
// entries are its distinct (j, n_ij - m_i) pairs (deduplicated through a
// shared-memory hash table) and the tile lists hold 16-bit entry numbers.
// Images are stored as 8-bit signed numbers per axis.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t img_code(int a, int b, int c) {
    return (uint32_t)(a + 128) | ((uint32_t)(b + 128) << 8) | ((uint32_t)(c + 128) << 16);
}

__device__ __forceinline__ float round_ratio(float num, float inv) {
    const float kShift = 12582912.0f;
    return __fsub_rn(__fmaf_rn(num, inv, kShift), kShift);
}

__device__ __forceinline__ uint32_t hash_slot(unsigned long long key) {
    return (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> 52) & (TILE_HASH - 1);
}

constexpr unsigned long long HASH_EMPTY = ~0ull;

template <int ND>
__global__ void __launch_bounds__(TILE_ATOMS) k_tile(DevCtx c, int all) {
    __shared__ unsigned long long hkey[TILE_HASH];
    __shared__ uint16_t hidx[TILE_HASH];
    __shared__ uint32_t wsum[TILE_ATOMS / 32];
    const uint32_t t = blockIdx.x;
    if (t >= c.ntile) return;
    const uint32_t s = c.tile_sys[t];
    if (!all && !c.flag[s]) return;
    const SysConst& S = c.sys[s];
    const uint32_t a0 = c.tile_atom0[t], na = c.tile_natom[t];
    const uint32_t tid = threadIdx.x;
    for (uint32_t q = tid; q < TILE_HASH; q += blockDim.x) hkey[q] = HASH_EMPTY;
    const float4 A0 = c.pos[2 * (size_t)a0];
    __syncthreads();
    const uint32_t i = a0 + tid;
    const bool act = tid < na && c.rank[i] != NOT_MEMBER;
    int m[3] = {0, 0, 0};
    uint32_t nn = 0;
    bool bad = false;
    float4 Ai = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act) {
        Ai = c.pos[2 * (size_t)i];
        m[0] = (int)round_ratio(Ai.x - A0.x, S.invLf[0]);
        m[1] = (int)round_ratio(Ai.y - A0.y, S.invLf[1]);
        if (ND == 3) m[2] = (int)round_ratio(Ai.z - A0.z, S.invLf[2]);
        nn = c.nnb[i];
        for (uint32_t k = 0; k < nn; k++) {
            const uint32_t j = c.nbr[(size_t)i * c.maxnb + k];
            const float4 Aj = c.pos[2 * (size_t)j];
            int im[3] = {0, 0, 0};
            im[0] = (int)round_ratio(Ai.x - Aj.x, S.invLf[0]) - m[0];
            im[1] = (int)round_ratio(Ai.y - Aj.y, S.invLf[1]) - m[1];
            if (ND == 3) im[2] = (int)round_ratio(Ai.z - Aj.z, S.invLf[2]) - m[2];
            if (im[0] < -127 || im[0] > 127 || im[1] < -127 || im[1] > 127 || im[2] < -127 || im[2] > 127)
                bad = true;
            const unsigned long long key = ((unsigned long long)j << 24) | img_code(im[0], im[1], im[2]);
            uint32_t slot = hash_slot(key);
            bool placed = false;
            for (uint32_t p = 0; p < TILE_HASH; p++) {   // bounded linear probing
                const unsigned long long old = atomicCAS(&hkey[slot], HASH_EMPTY, key);
                if (old == HASH_EMPTY || old == key) {
                    placed = true;
                    break;
                }
                slot = (slot + 1) & (TILE_HASH - 1);
            }
            if (!placed) bad = true;
        }
        if (m[0] < -127 || m[0] > 127 || m[1] < -127 || m[1] > 127 || m[2] < -127 || m[2] > 127) bad = true;
        c.atom_img[i] = img_code(m[0], m[1], m[2]);
    }
    if (bad) atomicOr(c.status, ST_IMAGE_RANGE | ST_TILE_OVERFLOW);
    __syncthreads();
    // compact the occupied slots into entry numbers (block exclusive scan)
    constexpr uint32_t PER = TILE_HASH / TILE_ATOMS;
    uint32_t cnt = 0;
    for (uint32_t q = 0; q < PER; q++) cnt += hkey[tid * PER + q] != HASH_EMPTY;
    const uint32_t lane = tid & 31u, warp = tid >> 5;
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t base = incl - cnt;
    for (uint32_t w = 0; w < warp; w++) base += wsum[w];
    uint32_t total = 0;
    for (uint32_t w = 0; w < TILE_ATOMS / 32; w++) total += wsum[w];
    for (uint32_t q = 0; q < PER; q++) {
        const uint32_t slot = tid * PER + q;
        const unsigned long long key = hkey[slot];
        if (key == HASH_EMPTY) continue;
        if (base < TILE_ECAP) c.tile_ent[(size_t)t * TILE_ECAP + base] = key;
        hidx[slot] = (uint16_t)min(base, (uint32_t)TILE_ECAP - 1u);
        base++;
    }
    if (tid == 0) {
        c.tile_ne[t] = min(total, (uint32_t)TILE_ECAP);
        c.tile_anchor[t] = A0;
        if (total > TILE_ECAP) atomicOr(c.status, ST_TILE_OVERFLOW);
    }
    __syncthreads();
    // tile lists: entry number of every (atom, neighbour)
    if (act) {
        uint16_t* lst = c.tile_lst + (size_t)t * c.maxnb * TILE_ATOMS + tid;
        for (uint32_t k = 0; k < nn; k++) {
            const uint32_t j = c.nbr[(size_t)i * c.maxnb + k];
            const float4 Aj = c.pos[2 * (size_t)j];
            int im[3] = {0, 0, 0};
            im[0] = (int)round_ratio(Ai.x - Aj.x, S.invLf[0]) - m[0];
            im[1] = (int)round_ratio(Ai.y - Aj.y, S.invLf[1]) - m[1];
            if (ND == 3) im[2] = (int)round_ratio(Ai.z - Aj.z, S.invLf[2]) - m[2];
            const unsigned long long key = ((unsigned long long)j << 24) | img_code(im[0], im[1], im[2]);
            uint32_t slot = hash_slot(key);
            uint16_t e = 0;
            for (uint32_t p = 0; p < TILE_HASH; p++) {
                const unsigned long long kk = hkey[slot];
                if (kk == key) {
                    e = hidx[slot];
                    break;
                }
                if (kk == HASH_EMPTY) break;
                slot = (slot + 1) & (TILE_HASH - 1);
            }
            lst[(size_t)k * TILE_ATOMS] = e;
        }
    }
}

// FP64 path: order each list by neighbour-list rank, which reproduces the
// reference's summation order (pairs (i, j<i) in ascending j, then (i'>i, i)
// in ascending i').
// The place of an entry is the number of entries with ranks below its own.
// Entries of smaller rank than the atom's come first; with pair slots
// (c.pairf), the CTA hands each list as many consecutive slots of its system.
constexpr uint32_t SORT_CAP = 256;   // longer lists are reported, not sorted
constexpr uint32_t SORT_WARPS = 8, SORT_SLOTS = 3;

// One list by one warp: the ranks are staged in shared memory and every lane
// counts for its entries (three of a list of up to 96).  A thread that
// insertion-sorted its own list kept both arrays in local memory and moved
// ~n^2/4 entries there: 268 -> 7.5 us at 1000 LJ atoms, 427 -> 31 us at 29,667,
// 7.57 -> 0.89 ms at 1,048,576 (~72 entries; one GB300).  All arguments are
// uniform in the warp; returns the number of entries ranked before the atom.
__device__ __forceinline__ uint32_t sort_list(const DevCtx& c, uint32_t i, uint32_t cnt, uint32_t lane, uint32_t* rk,
                                              uint32_t* jv) {
    if (!cnt) return 0u;
    uint32_t* row = c.nbr + (size_t)i * c.maxnb;
    const uint32_t ri = c.rank[i];
    const uint32_t padded = (cnt + 3u) & ~3u;   // <= SORT_CAP
    uint32_t below = 0u;
    for (uint32_t q = lane; q < padded; q += 32u) {
        const uint32_t j = q < cnt ? row[q] : 0u;
        const uint32_t r = q < cnt ? c.rank[j] : 0xFFFFFFFFu;
        jv[q] = j;
        rk[q] = r;
        below += r < ri ? 1u : 0u;
    }
    below = __reduce_add_sync(0xFFFFFFFFu, below);
    __syncwarp();
    for (uint32_t q0 = 0; q0 < cnt; q0 += 32u * SORT_SLOTS) {
        uint32_t mine[SORT_SLOTS], pos[SORT_SLOTS];
#pragma unroll
        for (uint32_t u = 0; u < SORT_SLOTS; u++) {
            const uint32_t q = q0 + lane + 32u * u;
            mine[u] = q < cnt ? rk[q] : 0u;
            pos[u] = 0u;
        }
#pragma unroll 2
        for (uint32_t t = 0; t < padded; t += 4u) {
            const uint4 K = *reinterpret_cast<const uint4*>(&rk[t]);
#pragma unroll
            for (uint32_t u = 0; u < SORT_SLOTS; u++)
                pos[u] += (K.x < mine[u] ? 1u : 0u) + (K.y < mine[u] ? 1u : 0u) + (K.z < mine[u] ? 1u : 0u) +
                          (K.w < mine[u] ? 1u : 0u);
        }
#pragma unroll
        for (uint32_t u = 0; u < SORT_SLOTS; u++) {
            const uint32_t q = q0 + lane + 32u * u;
            if (q < cnt) row[pos[u]] = jv[q];
        }
    }
    return below;
}

// LANES lanes per list.  Eight, for lists of a few entries: where none of a
// warp's four lists is longer than four entries a lane, entries and ranks stay
// in registers; else the warp takes its lists one after the other.  With a warp
// per list / eight lanes: 400,000 disks with lists of 2.3 / 10 / 23 entries 123
// / 28, 140 / 37, 172 / 72 us, 65,536 disks (5 entries) 24 / 8.5 us, 48 WCA
// replicas (7) 143 / 33 us, 5003 spheres 4.9 / 5.0 us; 1000 and 29,667 LJ atoms
// (80) 6.4 / 14 and 34 / 37 us.
template <uint32_t LANES>
__global__ void __launch_bounds__(SORT_WARPS * 32) k_sort_lists(DevCtx c, int all) {
    constexpr uint32_t LISTS = SORT_WARPS * 32u / LANES, GROUPS = 32u / LANES, EACH = 4;
    static_assert(LISTS <= 32, "one warp hands out the slots");
    __shared__ __align__(16) uint32_t rk[SORT_WARPS][SORT_CAP], jv[SORT_WARPS][SORT_CAP];
    __shared__ uint32_t low[LISTS], sysw[LISTS];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t gl = lane % LANES, group = lane / LANES, list = threadIdx.x / LANES;
    const uint32_t i = blockIdx.x * LISTS + list;   // uniform in the group from here
    const uint32_t s = i < c.n ? c.atom_sys[i] : 0u;
    const bool go = i < c.n && (all || c.flag[s]);
    uint32_t cnt = go ? min(c.nnb[i], c.maxnb) : 0u;
    if (cnt > SORT_CAP) {
        if (gl == 0) atomicOr(c.status, ST_SORT_CAP);
        cnt = 0u;
    }
    uint32_t below = 0u;
    const uint32_t most = LANES == 32u ? cnt : __reduce_max_sync(0xFFFFFFFFu, cnt);   // uniform in the warp
    if (LANES < 32u && most <= EACH * LANES) {
        uint32_t* row = c.nbr + (size_t)i * c.maxnb;
        const uint32_t ri = cnt ? c.rank[i] : 0u;
        uint32_t j[EACH], r[EACH], pos[EACH];
#pragma unroll
        for (uint32_t u = 0; u < EACH; u++) {
            const uint32_t q = gl + LANES * u;
            j[u] = q < cnt ? row[q] : 0u;
            pos[u] = 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < EACH; u++) {
            r[u] = gl + LANES * u < cnt ? c.rank[j[u]] : 0xFFFFFFFFu;
            below += r[u] < ri ? 1u : 0u;
        }
#pragma unroll
        for (uint32_t v = 0; v < EACH; v++) {
            if (LANES * v >= most) break;
            for (uint32_t t = 0; t < min(LANES, most - LANES * v); t++) {
                const uint32_t k = __shfl_sync(0xFFFFFFFFu, r[v], t, LANES);
#pragma unroll
                for (uint32_t u = 0; u < EACH; u++) pos[u] += k < r[u] ? 1u : 0u;
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < EACH; u++)
            if (gl + LANES * u < cnt) row[pos[u]] = j[u];
#pragma unroll
        for (uint32_t o = LANES / 2; o; o >>= 1) below += __shfl_xor_sync(0xFFFFFFFFu, below, o, LANES);
    } else if (LANES == 32u) {
        below = sort_list(c, i, cnt, lane, rk[w], jv[w]);
    } else {
        for (uint32_t g = 0; g < GROUPS; g++) {
            const uint32_t ig = __shfl_sync(0xFFFFFFFFu, i, g * LANES), cg = __shfl_sync(0xFFFFFFFFu, cnt, g * LANES);
            const uint32_t bg = sort_list(c, ig, cg, lane, rk[w], jv[w]);
            __syncwarp();
            if (group == g) below = bg;
        }
    }
    if (!c.pairf) return;
    if (gl == 0) {
        low[list] = below;
        sysw[list] = go ? s : 0xFFFFFFFFu;
    }
    __syncthreads();
    // warp 0, all of its lanes: one atomic per system with lists in the CTA
    if (w != 0) return;
    constexpr uint32_t NONE = 0xFFFFFFFFu;
    const uint32_t my = lane < LISTS ? sysw[lane] : NONE;
    uint32_t before = 0u, total = 0u, leader = lane;
    for (uint32_t k = 0; k < LISTS; k++) {
        if (sysw[k] == my) {
            leader = min(leader, k);
            total += low[k];
            if (k < lane) before += low[k];
        }
    }
    uint32_t first = 0u;
    if (my != NONE && leader == lane) first = atomicAdd(&c.half_cnt[my], total);
    first = __shfl_sync(0xFFFFFFFFu, first, leader);
    if (my == NONE) return;
    const uint32_t me = blockIdx.x * LISTS + lane;
    // lists cut at their capacity (reported) need not be symmetric: never past the system's slots
    const bool fits = (size_t)first + before + low[lane] <= (size_t)c.sys[my].natoms * c.maxnb / 2;
    c.half_n[me] = fits ? low[lane] : 0u;
    c.half_base[me] = (uint32_t)((size_t)c.sys[my].atom_off * c.maxnb / 2) + first + before;
}

// slots of the pairs that an atom is second in: its place in the first atom's
// list, by bisection of that (sorted) list
__global__ void __launch_bounds__(BLOCK) k_slots(DevCtx c, int all) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i = blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5);
    if (i >= c.n || !(all || c.flag[c.atom_sys[i]])) return;
    const uint32_t cnt = min(c.nnb[i], c.maxnb), ri = c.rank[i];
    for (uint32_t k = c.half_n[i] + lane; k < cnt; k += 32u) {
        const uint32_t j = c.nbr[(size_t)i * c.maxnb + k];
        const uint32_t* row = c.nbr + (size_t)j * c.maxnb;
        uint32_t lo = 0, hi = c.half_n[j];   // first entry whose rank is not below ri
        const uint32_t nj = hi;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (c.rank[row[mid]] < ri) lo = mid + 1; else hi = mid;
        }
        // not found only in lists that are about to be rebuilt (a capacity cut)
        c.slots[(size_t)i * c.maxnb + k] = (lo < nj && row[lo] == i) ? c.half_base[j] + lo : NO_SLOT;
    }
}

void launch_half(const DevCtx& c, cudaStream_t s, int all) {
    if (all && c.pairf) cudaMemsetAsync(c.half_cnt, 0, 4 * (size_t)c.nsys, s);
    if (c.list_mean <= 24u) k_sort_lists<8><<<grid_for(c.n, SORT_WARPS * 4), SORT_WARPS * 32, 0, s>>>(c, all);
    else k_sort_lists<32><<<grid_for(c.n, SORT_WARPS), SORT_WARPS * 32, 0, s>>>(c, all);
    if (c.pairf) k_slots<<<grid_for(c.n, BLOCK / 32), BLOCK, 0, s>>>(c, all);
}

// ---------------------------------------------------------------------------
// explicit rebuild test (NeighborList::update(false) outside a time step)
// ---------------------------------------------------------------------------
template <int ND>
__global__ void k_check(DevCtx c) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = false;
    double dsq = 0.0;
    uint32_t s = 0;
    if (i < c.n) {
        s = c.atom_sys[i];
        if (c.rank[i] != NOT_MEMBER) {
            dsq = disp_sq<ND>(ldx<ND>(c.x, i), ldx<ND>(c.lastloc, i));
            valid = !(dsq != dsq);
        }
    }
    check_accumulate(c, s, valid, dsq);
}

// number of half-list pairs per atom (neighbours with smaller rank)
__global__ void k_count_half(DevCtx c) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    uint32_t ri = c.rank[i];
    uint32_t cnt = 0;
    if (ri != NOT_MEMBER) {
        uint32_t nn = c.nnb[i];
        for (uint32_t k = 0; k < nn; k++)
            if (c.rank[c.nbr[(size_t)i * c.maxnb + k]] < ri) cnt++;
    }
    c.red[i] = (double)cnt;
}

template <int ND>
__global__ void k_posq(DevCtx c) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    using V = typename DVec<ND>::T;
    V xk = static_cast<const V*>(c.x)[k];
    const double* xs = reinterpret_cast<const double*>(&xk);
    float4 A, B;
    posq_split(xs[0], A.x, B.x);
    posq_split(xs[1], A.y, B.y);
    if constexpr (ND == 3) posq_split(xs[2], A.z, B.z); else { A.z = 0.f; B.z = 0.f; }
    A.w = (float)c.diam[k];
    B.w = 0.f;
    c.pos[2 * (size_t)(k)] = A;
    c.pos[2 * (size_t)(k) + 1] = B;
    if (c.staged) c.rec[k] = make_record(A, B, c.rframe[k]);
}

// the cell-block records of every atom in the frames of the current cells
// (after a box change on the same cell grids, or when the mixed path moves to
// the cell-block kernels between list builds)
template <int ND>
__global__ void k_reframe(DevCtx c) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    const uint32_t s = c.atom_sys[k];
    float4 A, B;
    ld_pos(c.pos, k, A, B);
    float4 fr = make_float4(0.f, 0.f, 0.f, __uint_as_float(REC_BIAS | (REC_BIAS << 12) | (REC_BIAS << 22)));
    if (c.rank[k] != NOT_MEMBER) {
        const SysConst& S = c.sys[s];
        uint32_t ci[3];
        cell_coords(S, c.bucket[k] - c.bucket_off[s], ci);
        bool ok;
        fr = rec_frame<ND>(S, ci, A, B, ok);
    }
    c.rframe[k] = fr;
    c.rec[k] = make_record(A, B, fr);
}

// ---------------------------------------------------------------------------
void launch_tiles(const DevCtx& c, cudaStream_t s, int all);

void launch_arm(const DevCtx& c, cudaStream_t s, int count_step, int use_cond,
                unsigned long long handle) {
    const unsigned threads = c.nsys <= 32 ? 32u : (c.nsys <= 256 ? 256u : 1024u);
    k_arm<<<1, threads, 0, s>>>(c, count_step, use_cond, (cudaGraphConditionalHandle)handle);
}

template <int ND>
static void sortgather(const DevCtx& c, cudaStream_t s) {
    // warps per cell: one per 32 atoms of the system of the fullest cells, at most
    // eight where other systems' cells alone give every SM its warps
    const uint32_t parts = std::max(1u, std::min((c.cell_mean + 31u) / 32u, std::max(8u, 152u * 32u / c.nbucket)));
    const auto grid = [&](uint32_t lanes) { return (unsigned)(((size_t)c.nbucket * parts * lanes + BLOCK - 1) / BLOCK); };
    // lanes per cell: a warp where cells hold more than eight atoms or a warp each
    // does not fill the SMs, else eight lanes, or four where eight for each cell
    // would fill the SMs more than once; sixteen where a few large cells among them
    // would otherwise be what all wait for
    const uint32_t mean = c.n / c.nbucket + 1u;
    if (mean > 8u || c.nbucket < 152u * 32u) k_sortgather<ND, 32><<<grid(32), BLOCK, 0, s>>>(c, parts);
    else if (c.cell_mean > 32u && c.nbucket < 20000u) k_sortgather<ND, 16><<<grid(16), BLOCK, 0, s>>>(c, parts);
    else if (mean > 4u || c.nbucket < 40000u) k_sortgather<ND, 8><<<grid(8), BLOCK, 0, s>>>(c, parts);
    else k_sortgather<ND, 4><<<grid(4), BLOCK, 0, s>>>(c, parts);
}

void launch_rebuild(const DevCtx& c, cudaStream_t s) {
    unsigned ga = grid_for(c.n);
    if (c.nd == 3) k_bin<3><<<ga, BLOCK, 0, s>>>(c); else k_bin<2><<<ga, BLOCK, 0, s>>>(c);
    const uint32_t nblk = (c.nbucket + SCAN_CHUNK - 1) / SCAN_CHUNK;
    if (nblk <= SCAN_ONE) {
        k_scan_one<<<1, SCAN_THREADS, 0, s>>>(c);
    } else {
        k_scan_blocks<<<nblk, SCAN_THREADS, 0, s>>>(c);
        k_scan_write<<<nblk, SCAN_THREADS, 0, s>>>(c);
    }
    if (c.nd == 3) {
        k_scatter<3><<<ga, BLOCK, 0, s>>>(c);
        sortgather<3>(c, s);
    } else {
        k_scatter<2><<<ga, BLOCK, 0, s>>>(c);
        sortgather<2>(c, s);
    }
    if (c.staged) {
        if (c.nd == 3) {
            k_copyback<3, true><<<ga, BLOCK, 0, s>>>(c);
        } else {
            k_copyback<2, true><<<ga, BLOCK, 0, s>>>(c);
        }
        launch_build_stg(c, s);
        return;
    }
    if (c.any_lees) {   // FP64 handles only
        if (c.nd == 3) {
            k_copyback<3, false><<<ga, BLOCK, 0, s>>>(c);
            k_build_lees<3><<<ga, BLOCK, 0, s>>>(c);
        } else {
            k_copyback<2, false><<<ga, BLOCK, 0, s>>>(c);
            k_build_lees<2><<<ga, BLOCK, 0, s>>>(c);
        }
        launch_half(c, s, 0);
        return;
    }
    // home atoms per warp: 32 (most cells whole) where the cells alone give every
    // SM its warps, shared among a few where some system's cells hold many more;
    // else as few as it takes to give every SM its warps
    const uint32_t want = 152u * 32u, mean = c.n / c.nbucket + 1u;
    uint32_t parts = std::min(std::max(want / c.nbucket, 1u), std::min(mean, 32u));
    const uint32_t per = parts == 1u ? 32u : std::min(32u, (mean + parts - 1u) / parts);
    if (c.cell_mean > 48u) parts = std::max(parts, std::min(8u, (c.cell_mean + 31u) / 32u));
    const unsigned gb = (unsigned)(((size_t)c.nbucket * parts + BUILD_WARPS - 1) / BUILD_WARPS);
    if (c.nd == 3) {
        k_copyback<3, false><<<ga, BLOCK, 0, s>>>(c);
        if (c.any_wrap) k_build<3, true><<<gb, BUILD_WARPS * 32, 0, s>>>(c, parts, per);
        else k_build<3, false><<<gb, BUILD_WARPS * 32, 0, s>>>(c, parts, per);
    } else {
        k_copyback<2, false><<<ga, BLOCK, 0, s>>>(c);
        if (c.any_wrap) k_build<2, true><<<gb, BUILD_WARPS * 32, 0, s>>>(c, parts, per);
        else k_build<2, false><<<gb, BUILD_WARPS * 32, 0, s>>>(c, parts, per);
    }
    if (c.prec == PREC_FP64) {
        launch_half(c, s, 0);
    } else if (c.ntile && c.tiled) {
        launch_tiles(c, s, 0);
    }
}

void launch_tiles(const DevCtx& c, cudaStream_t s, int all) {
    if (c.nd == 3) k_tile<3><<<c.ntile, TILE_ATOMS, 0, s>>>(c, all);
    else k_tile<2><<<c.ntile, TILE_ATOMS, 0, s>>>(c, all);
}

void launch_check(const DevCtx& c, cudaStream_t s) {
    if (c.nd == 3) k_check<3><<<grid_for(c.n), BLOCK, 0, s>>>(c);
    else k_check<2><<<grid_for(c.n), BLOCK, 0, s>>>(c);
}

void launch_numpairs(const DevCtx& c, cudaStream_t s) {
    k_count_half<<<grid_for(c.n), BLOCK, 0, s>>>(c);
}

void launch_reframe(const DevCtx& c, cudaStream_t s) {
    if (!c.rec) return;
    if (c.nd == 3) k_reframe<3><<<grid_for(c.n), BLOCK, 0, s>>>(c);
    else k_reframe<2><<<grid_for(c.n), BLOCK, 0, s>>>(c);
}

void launch_posq(const DevCtx& c, cudaStream_t s) {
    if (c.nd == 3) k_posq<3><<<grid_for(c.n), BLOCK, 0, s>>>(c);
    else k_posq<2><<<grid_for(c.n), BLOCK, 0, s>>>(c);
}

// ---------------------------------------------------------------------------
__global__ void k_remainder_test(const double* d, const double* L, double* out, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double l = L[i];
    out[i] = remainder_exact(d[i], l, 1.0 / l, 0.5 * l);
}

void launch_remainder_test(const double* d, const double* L, double* out, uint32_t n,
                           cudaStream_t s) {
    k_remainder_test<<<grid_for(n), BLOCK, 0, s>>>(d, L, out, n);
}

}  // namespace parm
