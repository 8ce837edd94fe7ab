// What the mixed-precision cell-block kernels share (staged.cu: list build, pair
// forces, list expansion; staged_eval.cu: energies and stresses): block tables,
// staging of a block's neighbourhood in shared memory, displacements.
//
// Reference behaviour (wackywendell/parm): NeighborList::update_list
// (src/trackers.cpp:19-85) keeps every pair with
// |diff(x_i, x_j)| < (d_i + d_j)/2 + skin; NListed::set_forces
// (src/interaction.hpp:2165-2175) adds the pair force of every listed pair.
// The pair set here is the reference's exactly (FP32 screening, exact FP64
// test near the threshold); forces are FP32 sums, as in pair32.cu.
//
// Blocks.  A system whose cell grid has at least 3 cells along every axis is
// cut into blocks of Kx x Ky cells of one z layer (x fastest, the order of
// the cells in memory).  The block's neighbourhood is made of "rows": the
// cells x0-1 .. x1 of the y rows y0-1 .. y1 in the z layers z-1, z, z+1
// (2D: no z).  Each row is three "pieces" (left cell, the block's own cells,
// right cell), each a contiguous range of atoms in memory with one periodic
// image; pieces are numbered row by row and their atoms get consecutive local
// indices.  Kx <= nx - 2 and Ky <= ny - 2, so no atom appears twice in a
// block's neighbourhood.
//
// Staged record (16 bytes) of atom j: its cell-block record (kept per atom
// by the list build and the time-step kernels; parm_ctx.cuh) moved into the
// block's frame.  The block frame's origin is the lower edge of its first
// neighbour cell along each axis (on the 1/8 grid); a piece adds one packed
// constant K_p (its periodic shift and, along y and z, its row origin, in
// units of 1/8) to the coarse fields and its periodic shift's fine part
// s (L - L8) to the fine part.  Every staged field is then an exact integer
// 8 * (local position) + 256 within [0, 3840) (x, 12 bits) or [0, 768)
// (y, z, 10 bits), and a pair displacement is 0.125 * (q_i - q_j) +
// (f_i - f_j): the coarse difference is exact and only the fine parts round.
// One 32-bit subtraction (W_i + 256 per field) - W_j forms the three biased
// differences at once (each in [0, 2^bits) for atoms less than 32 apart, so
// no borrow crosses a field), and OR-ing a field into the mantissa of
// 1.5 * 2^20 (ulp 1/8) turns it into 1.5 * 2^20 + (q_i - q_j + 256) / 8
// exactly.
//
// The list build only screens candidates, so it stages plain FP32 positions
// relative to the centre of the block's neighbourhood (0.125 (q - c) + f, one
// rounding); pairs within 2e-5 (relative, on r^2) of the threshold are
// decided by the exact FP64 test.
//
// Lists.  Entries are 16-bit local indices.  The home atoms of a block are the
// atoms of its own pieces in the z = 0 layer (one contiguous range of memory
// per home row).  For a home row starting at atom s0 with H atoms, entry k of
// home atom s0 + h lives at u16 offset s0 * maxnb + (k / 2) * 2H + 2h + k % 2,
// so a warp reads the entries of 32 consecutive atoms as one coalesced line of
// 32-bit words (two entries each).
#pragma once
#include "fpbits.cuh"
#include "parm_check.cuh"
#include "parm_pair32.cuh"

namespace parm {

constexpr int STG_THREADS = STG_THREADS_HOST;
constexpr float STG_BAND = 2e-5f;   // relative band on r^2 decided by the exact FP64 test
constexpr float CUT_BAND_S = 4e-6f; // LJ cut-off band (see pair32.cu)

struct __align__(16) StgTable {
    uint32_t g0[STG_PIECES_MAX];        // first atom of each piece
    uint32_t cnt[STG_PIECES_MAX];       // atoms in each piece
    uint32_t off[STG_PIECES_MAX + 1];   // local index of the first atom of each piece
    uint32_t K[STG_PIECES_MAX];         // packed coarse shift of each piece
    float F[STG_PIECES_MAX][3];         // fine part of each piece's periodic shift
    uint32_t rowbase[STG_ROWS_MAX];     // bucket of cell x = 0 of each row
    uint32_t hoff[STG_KY_MAX + 1];      // home atoms before each home row
    uint32_t hnmax[STG_KY_MAX];         // longest list of each home row (from the last build)
    int pc[3];                          // 256 + 8 * (neighbourhood centre) (plain positions)
    uint32_t nrow, npiece, total, nhome, nyr;
    int x0, x1, y0, y1, z;
};

static_assert(sizeof(StgTable) <= 16 * STG_TAB_WORDS, "block table larger than its slot");
constexpr uint32_t STG_TAB_USED = (uint32_t)((sizeof(StgTable) + 15) / 16);

__device__ __forceinline__ int wrap_idx(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// The block tables depend on the cell arrays and the box only: the list
// build (and the list conversion) store them, the per-step kernels load them.
__device__ __forceinline__ void stg_store_table(const DevCtx& c, const StgTable& T, uint32_t b) {
    const float4* src = reinterpret_cast<const float4*>(&T);
    for (uint32_t t = threadIdx.x; t < STG_TAB_USED; t += blockDim.x)
        c.stg_tab[(size_t)b * STG_TAB_WORDS + t] = src[t];
}
// longest list of each home row (all threads; ends with a barrier)
template <int ND>
__device__ void stg_row_nmax(const DevCtx& c, StgTable& T) {
    for (uint32_t r = threadIdx.x; r < STG_KY_MAX; r += blockDim.x) T.hnmax[r] = 0u;
    __syncthreads();
    for (uint32_t h = threadIdx.x; h < T.nhome; h += blockDim.x) {
        uint32_t hr = 0;
        while (h >= T.hoff[hr + 1]) hr++;
        const uint32_t p = 3u * ((ND == 3 ? T.nyr : 0u) + hr + 1u) + 1u;
        atomicMax(&T.hnmax[hr], c.nnb[T.g0[p] + (h - T.hoff[hr])]);
    }
    __syncthreads();
}

__device__ __forceinline__ void stg_load_table(const DevCtx& c, StgTable& T, uint32_t b) {
    float4* dst = reinterpret_cast<float4*>(&T);
    for (uint32_t t = threadIdx.x; t < STG_TAB_USED; t += blockDim.x)
        dst[t] = __ldg(&c.stg_tab[(size_t)b * STG_TAB_WORDS + t]);
    __syncthreads();
}

// fill the block table (all threads; ends with a barrier)
template <int ND>
__device__ void stg_setup(const DevCtx& c, const SysConst& S, const uint4& bd, StgTable& T) {
    const int x0 = (int)(bd.y & 0xFFFFu), x1 = (int)(bd.y >> 16);
    const int y0 = (int)(bd.z & 0xFFFFu), y1 = (int)(bd.z >> 16);
    const int z = (int)bd.w;
    const int nyr = y1 - y0 + 2;
    const int nrow = (ND == 3 ? 3 : 1) * nyr;
    const int npiece = 3 * nrow;
    const uint32_t b0 = c.bucket_off[bd.x];
    const int nx = S.nc[0], ny = S.nc[1], nz = S.nc[2];
    // block frame origin (units of 1/8): lower edge of the first neighbour cell
    const int xb8 = rec_origin8(S, 0, x0 - 1), yb8 = rec_origin8(S, 1, y0 - 1);
    const int zb8 = (ND == 3) ? rec_origin8(S, 2, z - 1) : 0;
    // one thread per piece (row r = t / 3, part t % 3: left cell, the block's
    // cells, right cell)
    for (int t = threadIdx.x; t < npiece; t += blockDim.x) {
        const int r = t / 3, part = t % 3;
        const int dz = (ND == 3) ? r / nyr - 1 : 0;
        const int yy = y0 - 1 + r % nyr, zz = z + dz;
        const int cy = wrap_idx(yy, ny), cz = (ND == 3) ? wrap_idx(zz, nz) : 0;
        const uint32_t rb = b0 + (uint32_t)((cz * ny + cy) * nx);
        if (part == 0) T.rowbase[r] = rb;
        uint32_t lo, hi;
        int sx = 0;   // periodic shift of the piece along x (boxes)
        if (part == 0) {
            lo = rb + (uint32_t)wrap_idx(x0 - 1, nx);
            hi = lo + 1;
            sx = x0 == 0 ? -1 : 0;
        } else if (part == 1) {
            lo = rb + (uint32_t)x0;
            hi = rb + (uint32_t)x1;
        } else {
            lo = rb + (uint32_t)wrap_idx(x1, nx);
            hi = lo + 1;
            sx = x1 == nx ? 1 : 0;
        }
        const int sy = yy < 0 ? -1 : (yy >= ny ? 1 : 0);
        const int sz = (ND == 3) ? (zz < 0 ? -1 : (zz >= nz ? 1 : 0)) : 0;
        const uint32_t g = c.cell_start[lo];
        T.g0[t] = g;
        T.cnt[t] = c.cell_start[hi] - g;
        const int kx = sx * (int)(S.L8[0] * 8.0f) - xb8;
        const int ky = rec_origin8(S, 1, cy) + sy * (int)(S.L8[1] * 8.0f) - yb8;
        const int kz = (ND == 3) ? rec_origin8(S, 2, cz) + sz * (int)(S.L8[2] * 8.0f) - zb8 : 0;
        T.K[t] = (uint32_t)kx + ((uint32_t)ky << 12) + ((uint32_t)kz << 22);
        T.F[t][0] = (float)sx * S.Lr8[0];
        T.F[t][1] = (float)sy * S.Lr8[1];
        T.F[t][2] = (float)sz * S.Lr8[2];
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        // exclusive scan of the piece sizes, 32 pieces per pass
        const uint32_t lane = threadIdx.x;
        uint32_t carry = 0;
        for (int base = 0; base < npiece; base += 32) {
            const int p = base + (int)lane;
            const uint32_t v = p < npiece ? T.cnt[p] : 0u;
            uint32_t inc = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= (uint32_t)o) inc += u;
            }
            if (p < npiece) T.off[p] = carry + inc - v;
            carry += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
        if (lane == 0) {
            T.off[npiece] = carry;
            T.total = carry;
            T.nrow = (uint32_t)nrow;
            T.npiece = (uint32_t)npiece;
            T.nyr = (uint32_t)nyr;
            T.x0 = x0; T.x1 = x1; T.y0 = y0; T.y1 = y1; T.z = z;
            const int hbase = (ND == 3) ? nyr : 0;   // first home row (z layer 0, y = y0)
            uint32_t h = 0;
            for (int hr = 0; hr < y1 - y0; hr++) {
                T.hoff[hr] = h;
                h += T.cnt[3 * (hbase + hr + 1) + 1];
            }
            T.hoff[y1 - y0] = h;
            for (int r = 0; r < STG_KY_MAX; r++) T.hnmax[r] = 0u;
            T.nhome = h;
            // centre of the neighbourhood in the block frame (plain positions)
            T.pc[0] = REC_BIAS + (int)rint(4.0 * (double)(x1 - x0 + 2) * S.cellw[0]);
            T.pc[1] = REC_BIAS + (int)rint(4.0 * (double)(y1 - y0 + 2) * S.cellw[1]);
            T.pc[2] = REC_BIAS + ((ND == 3) ? (int)rint(12.0 * S.cellw[2]) : 0);
        }
    }
    __syncthreads();
}

// cell-block record R of an atom of piece p, moved into the block frame
__device__ __forceinline__ float4 stg_shift(const StgTable& T, uint32_t p, const float4& R) {
    return make_float4(R.x + T.F[p][0], R.y + T.F[p][1], R.z + T.F[p][2],
                       __uint_as_float(__float_as_uint(R.w) + T.K[p]));
}

// one bulk request that brings [p, p + bytes) into L2 (16-byte aligned start
// and size); it completes on its own and nothing waits for it
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// the records of the block's pieces (and, for the force kernel, the home
// rows' lists) requested into L2 at once, ahead of the staging loads
template <int ND>
__device__ __forceinline__ void stg_prefetch(const DevCtx& c, const StgTable& T, bool lists) {
    for (uint32_t t = threadIdx.x; t < T.npiece; t += blockDim.x)
        if (T.cnt[t]) prefetch_l2(c.rec + T.g0[t], T.cnt[t] * 16u);
    const uint32_t nhr = (uint32_t)(T.y1 - T.y0);
    if (lists && threadIdx.x >= 128u && threadIdx.x - 128u < nhr) {
        const uint32_t p = 3u * ((ND == 3 ? T.nyr : 0u) + (threadIdx.x - 128u) + 1u) + 1u;
        // the row's lists are word-major (word w of atom h at w * H + h), so
        // the words in use form a prefix; rows start 16-byte aligned (maxnb
        // is a multiple of 8) and the prefix is rounded up inside the row
        const uint32_t words = ((T.hnmax[threadIdx.x - 128u] + 1u) >> 1) * T.cnt[p];
        const uint32_t bytes = min((words * 4u + 15u) & ~15u, T.cnt[p] * c.maxnb * 2u);
        if (bytes) prefetch_l2(c.nbr16 + (size_t)T.g0[p] * c.maxnb, bytes);
    }
}

// piece of local index q (binary search over the offsets)
__device__ __forceinline__ uint32_t stg_piece(const StgTable& T, uint32_t q) {
    uint32_t lo = 0, hi = T.npiece;   // off[lo] <= q < off[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (T.off[mid] <= q) lo = mid; else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t stg_global(const StgTable& T, uint32_t q) {
    const uint32_t p = stg_piece(T, q);
    return T.g0[p] + (q - T.off[p]);
}

// a local index that does not belong to the block (inconsistent lists) is
// reported and replaced by the home atom itself, whose pair term is zero
__device__ __forceinline__ uint32_t stg_check(const DevCtx& c, const StgTable& T, uint32_t q, uint32_t qi) {
    if (q < T.total) return q;
    atomicOr(c.status, ST_TILE_OVERFLOW);
    return qi;
}

// record of local index q: shared memory, or rebuilt from global memory when
// the neighbourhood is larger than the staging capacity
template <int ND>
__device__ __forceinline__ float4 stg_get(const DevCtx& c, const SysConst& S, const StgTable& T,
                                          const float4* srec, uint32_t cap, uint32_t q) {
    if (q < cap) return srec[q];
    const uint32_t p = stg_piece(T, q);
    return stg_shift(T, p, c.rec[T.g0[p] + (q - T.off[p])]);
}

constexpr uint32_t STG_GUARD = 256u | (256u << 12) | (256u << 22);   // + 256 per field
constexpr uint32_t STG_MANT = 0x49C00000u;                           // 1.5 * 2^20, ulp 1/8
constexpr float STG_K = 1572864.0f + 32.0f;                          // 1.5 * 2^20 + 256 / 8

// W_i + 256 per field (the home atom's side of the packed subtraction)
__device__ __forceinline__ uint32_t stg_wi(const float4& ri) { return __float_as_uint(ri.w) + STG_GUARD; }

// displacement x_i - x_j from two packed records
template <int ND>
__device__ __forceinline__ void stg_disp(uint32_t wi, const float4& ri, const float4& rj, float* r) {
    const uint32_t D = wi - __float_as_uint(rj.w);
    r[0] = (__uint_as_float((D & 0xFFFu) | STG_MANT) - STG_K) + (ri.x - rj.x);
    r[1] = (__uint_as_float(((D >> 12) & 0x3FFu) | STG_MANT) - STG_K) + (ri.y - rj.y);
    if constexpr (ND == 3) r[2] = (__uint_as_float((D >> 22) | STG_MANT) - STG_K) + (ri.z - rj.z);
    else r[2] = 0.f;
}

// plain FP32 position relative to the neighbourhood centre (list screening)
__device__ __forceinline__ float4 stg_plain(const StgTable& T, const float4& rec, float w) {
    const uint32_t W = __float_as_uint(rec.w);
    const float qx = (float)((int)(W & 0xFFFu) - T.pc[0]), qy = (float)((int)((W >> 12) & 0x3FFu) - T.pc[1]),
                qz = (float)((int)(W >> 22) - T.pc[2]);
    return make_float4(fmaf(qx, 0.125f, rec.x), fmaf(qy, 0.125f, rec.y), fmaf(qz, 0.125f, rec.z), w);
}

// The plain stage is pair-interleaved: local indices 2k and 2k + 1 share 32
// bytes, (x0, x1, y0, y1) then (z0, z1, w0, w1), so one 16-byte load gives the
// x and y of two candidates as packed FP32 pairs.
__device__ __forceinline__ void stg_put_plain(float4* sp, uint32_t q, const float4& v) {
    float* f = reinterpret_cast<float*>(sp) + 8u * (q >> 1) + (q & 1u);
    f[0] = v.x;
    f[2] = v.y;
    f[4] = v.z;
    f[6] = v.w;
}
__device__ __forceinline__ float4 stg_at_plain(const float4* sp, uint32_t q) {
    const float* f = reinterpret_cast<const float*>(sp) + 8u * (q >> 1) + (q & 1u);
    return make_float4(f[0], f[2], f[4], f[6]);
}

// list diameter of atom j (the w of its coarse position view)
__device__ __forceinline__ float stg_diam(const DevCtx& c, uint32_t j) {
    return __ldg(reinterpret_cast<const float*>(c.pos + 2 * (size_t)j) + 3);
}

// Staging for the list build: plain FP32 positions of the first `cap` local
// indices (w: the list diameter when `diam`, else 0), warp per piece.  Each
// warp takes two pieces at a time and each lane issues the loads of up to
// four atoms (two per piece) before converting any, so that their latencies
// overlap.
static __device__ void stg_load_plain(const DevCtx& c, const StgTable& T, float4* sp, uint32_t cap, bool diam) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t p0 = warp; p0 < T.npiece; p0 += 2 * nw) {
        float4 R[4];
        float w[4];
        uint32_t q[4], pc[4];
        bool ok[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t p = p0 + (k >> 1) * nw;
            const uint32_t t = lane + 32u * (k & 1);
            pc[k] = p;
            ok[k] = p < T.npiece && t < T.cnt[p] && T.off[p] + t < cap;
            q[k] = ok[k] ? T.off[p] + t : 0u;
            w[k] = 0.f;
            if (ok[k]) {
                const uint32_t j = T.g0[p] + t;
                R[k] = __ldg(&c.rec[j]);
                if (diam) w[k] = stg_diam(c, j);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (ok[k]) stg_put_plain(sp, q[k], stg_plain(T, stg_shift(T, pc[k], R[k]), w[k]));
        // pieces longer than 64 atoms (large blocks of sparse systems)
#pragma unroll 1
        for (int k = 0; k < 2; k++) {
            const uint32_t p = p0 + k * nw;
            if (p >= T.npiece) break;
            for (uint32_t t = lane + 64u; t < T.cnt[p] && T.off[p] + t < cap; t += 32u) {
                const uint32_t j = T.g0[p] + t;
                stg_put_plain(sp, T.off[p] + t, stg_plain(T, stg_shift(T, p, __ldg(&c.rec[j])), diam ? stg_diam(c, j) : 0.f));
            }
        }
    }
    __syncthreads();
}

// ---- bulk (TMA) staging: one asynchronous copy per piece into shared memory,
// completion counted in bytes on one mbarrier ----
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}
// waits for phase 0 of the barrier, at most `limit` polls; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t limit) {
    for (uint32_t it = 0; it < limit; it++) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(0u)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Staging by bulk copies: every piece's records (and, EXTRA == 2, its FP32
// pair parameters) are copied into shared memory as they lie in global
// memory (one asynchronous copy per piece, 16-byte aligned, completion
// counted on one mbarrier), then each warp moves its pieces' records into
// the block frame in place.  Returns false (and flags ST_STAGE_TIMEOUT) when
// the copies do not complete within the wait limit; if they are still not
// complete after a second bounded wait, no thread touches the staged shared
// memory again.
template <int ND, int EXTRA>
__device__ bool stg_load_bulk(const DevCtx& c, const StgTable& T, float4* srec, void* sext, uint32_t cap,
                              uint64_t* bar) {
    const uint32_t staged = min(T.total, cap);
    const uint32_t per = (EXTRA == 2) ? 32u : 16u;
    if (threadIdx.x == 0) mbar_init(bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) mbar_arrive_tx(bar, staged * per);
    for (uint32_t p = threadIdx.x; p < T.npiece; p += blockDim.x) {
        const uint32_t o = T.off[p];
        if (o >= cap || T.cnt[p] == 0) continue;
        const uint32_t n = min(T.cnt[p], cap - o);
        bulk_g2s(srec + o, c.rec + T.g0[p], n * 16u, bar);
        if constexpr (EXTRA == 2) bulk_g2s(static_cast<float4*>(sext) + o, c.prm32 + T.g0[p], n * 16u, bar);
    }
    const bool ok = mbar_wait(bar, 1u << 22);
    bool settled = ok;
    if (!ok) {
        atomicOr(c.status, ST_STAGE_TIMEOUT);
        settled = mbar_wait(bar, 1u << 22);   // the copies in flight, once more with a limit
    }
    // unless every thread saw the copies complete, the block leaves its
    // shared memory alone (no rewrite, no pair loop) and returns at once
    if (!__syncthreads_and(settled)) return false;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t p = warp; p < T.npiece; p += nw) {
        const uint32_t o = T.off[p];
        if (o >= cap) continue;
        const uint32_t n = min(T.cnt[p], cap - o);
        const uint32_t K = T.K[p];
        const float F0 = T.F[p][0], F1 = T.F[p][1], F2 = T.F[p][2];
        for (uint32_t t = lane; t < n; t += 32u) {
            float4 r = srec[o + t];
            r.x += F0;
            r.y += F1;
            r.z += F2;
            r.w = __uint_as_float(__float_as_uint(r.w) + K);
            srec[o + t] = r;
            if constexpr (EXTRA == 1) static_cast<float*>(sext)[o + t] = __ldg(&c.prm32[T.g0[p] + t].y);
        }
    }
    return __syncthreads_and(ok) != 0;   // the same answer in every thread
}

// home atom h -> (home row, global atom, local index, cell x)
struct HomeAtom {
    uint32_t hr, i, qi, s0, H, hs;
    int cx;
};

template <int ND, bool CELL = true>
__device__ __forceinline__ HomeAtom stg_home(const DevCtx& c, const StgTable& T, uint32_t h) {
    HomeAtom a;
    uint32_t hr = 0;
    while (h >= T.hoff[hr + 1]) hr++;
    const uint32_t r = (ND == 3 ? T.nyr : 0u) + hr + 1u;
    const uint32_t p = 3u * r + 1u;
    a.hr = hr;
    a.hs = h - T.hoff[hr];
    a.s0 = T.g0[p];
    a.H = T.cnt[p];
    a.i = a.s0 + a.hs;
    a.qi = T.off[p] + a.hs;
    a.cx = T.x0;
    if constexpr (CELL) {
        a.cx = (int)(c.bucket[a.i] - T.rowbase[r]);
        if (a.cx < T.x0 || a.cx >= T.x1) {   // never for lists of the current grid
            atomicOr(c.status, ST_CELL_RANGE);
            a.cx = T.x0;
        }
    }
    return a;
}

// local candidate range of a home atom in stencil row r
__device__ __forceinline__ void stg_range(const DevCtx& c, const StgTable& T, uint32_t r, int cx,
                                          uint32_t& lo, uint32_t& hi) {
    const uint32_t pm = 3u * r + 1u;
    lo = (cx == T.x0) ? T.off[pm - 1] : T.off[pm] + (c.cell_start[T.rowbase[r] + (uint32_t)(cx - 1)] - T.g0[pm]);
    hi = (cx == T.x1 - 1) ? T.off[pm + 1] + T.cnt[pm + 1]   // through the right piece
                          : T.off[pm] + (c.cell_start[T.rowbase[r] + (uint32_t)(cx + 2)] - T.g0[pm]);
}

__device__ __forceinline__ size_t stg_entry16(const HomeAtom& a, uint32_t maxnb, uint32_t k) {
    return (size_t)a.s0 * maxnb + (size_t)(k >> 1) * 2u * a.H + 2u * a.hs + (k & 1u);
}

// exact reference list test, explicit round-to-nearest FP64 operations:
// diff(x_i, x_j).norm() < (d_i + d_j)/2 + skin
template <int ND>
__device__ __noinline__ bool keep_exact_rn(const DevCtx& c, const SysConst& S, uint32_t i, uint32_t j) {
    const double* a = reinterpret_cast<const double*>(c.x) + (size_t)i * (ND == 3 ? 4 : 2);
    const double* b = reinterpret_cast<const double*>(c.x) + (size_t)j * (ND == 3 ? 4 : 2);
    double sq[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int d = 0; d < ND; d++) {
        const double r = remainder_exact(__dsub_rn(a[d], b[d]), S.L[d], S.invL[d], S.halfL[d]);
        sq[d] = __dmul_rn(r, r);
    }
    double s2 = __dadd_rn(sq[0], sq[1]);
    if constexpr (ND == 3) s2 = __dadd_rn(s2, sq[2]);
    const double diam = __dmul_rn(__dadd_rn(c.diam[i], c.diam[j]), 0.5);
    return __dsqrt_rn(s2) < __dadd_rn(diam, S.skin);
}

__device__ __forceinline__ bool is_excluded_s(const DevCtx& c, uint32_t oi, uint32_t oj) {
    for (uint32_t e = c.excl_off[oi]; e < c.excl_off[oi + 1]; e++)
        if (c.excl_list[e] == oj) return true;
    return false;
}

// exact LJ cut-off classification (as lj_beyond_exact in pair32.cu)
static __device__ __noinline__ bool lj_beyond_exact_s(const DevCtx& c, const SysConst& S, uint32_t i, uint32_t j,
                                               int nd) {
    const double* xi = reinterpret_cast<const double*>(c.x) + (size_t)i * (nd == 3 ? 4 : 2);
    const double* xj = reinterpret_cast<const double*>(c.x) + (size_t)j * (nd == 3 ? 4 : 2);
    double sq[3] = {0.0, 0.0, 0.0};
    for (int d = 0; d < nd; d++) {
        double r = remainder_exact(__dsub_rn(xi[d], xj[d]), S.L[d], S.invL[d], S.halfL[d]);
        sq[d] = __dmul_rn(r, r);
    }
    double dsq = __dadd_rn(sq[0], sq[1]);
    if (nd == 3) dsq = __dadd_rn(dsq, sq[2]);
    const AtomPrm A = c.prm[i], B = c.prm[j];
    const double sig = __dmul_rn(__dadd_rn(A.p1, B.p1), 0.5);
    const double cut = B.p2 > A.p2 ? B.p2 : A.p2;
    const double rsq = __ddiv_rn(dsq, __dmul_rn(sig, sig));
    return rsq > __dmul_rn(cut, cut);
}

// non-member atoms of a system (no neighbours, zero force)
static __device__ void stg_nonmembers(const DevCtx& c, uint32_t s, int zero_a) {
    const SysConst& S = c.sys[s];
    const uint32_t b = c.bucket_off[s] + S.ncell;
    const uint32_t hi = S.atom_off + S.natoms;
    const uint32_t lo = max(c.cell_start[b], S.atom_off);
    for (uint32_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        c.nnb[i] = 0u;
        c.f32[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (zero_a) {
            double* a = static_cast<double*>(c.a) + (size_t)i * (c.nd == 3 ? 4 : 2);
            for (int d = 0; d < c.nd; d++) a[d] = 0.0;
        }
    }
}

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// packed pairs of FP32 values (Blackwell's f32x2 add / mul / fma: two lanes
// of work per instruction)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(f32x2 r, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

}  // namespace parm
