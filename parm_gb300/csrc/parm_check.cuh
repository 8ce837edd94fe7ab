// Per-system "two largest displacements" reduction used by the neighbour-list
// rebuild test (reference: NeighborList::update_list(false), trackers.cpp:23-53).
//
// Each atom contributes its squared FP64 displacement since the last list
// build.  The two largest values per system are kept as the bit patterns of
// non-negative doubles in `top[2s]` (largest) and `top[2s+1]` (second), which
// order like unsigned integers, so atomicMax reproduces the multiset top-2:
// a value that is displaced from the top slot is pushed into the second slot.
// Values are first reduced within a warp (and then a block) when all lanes
// belong to the same system, so a single large system costs two atomics per
// block.
#pragma once
#include "parm_ctx.cuh"

namespace parm {

__device__ __forceinline__ void top2_merge(unsigned long long& a1, unsigned long long& a2,
                                           unsigned long long b1, unsigned long long b2) {
    // merge (a1 >= a2) with (b1 >= b2) into the two largest of the four
    if (b1 > a1) {
        unsigned long long t = a1;
        a1 = b1;
        a2 = (t > b2) ? t : b2;
    } else {
        a2 = (b1 > a2) ? b1 : a2;
    }
}

__device__ __forceinline__ void top2_push(unsigned long long* top, unsigned long long t1,
                                          unsigned long long t2) {
    if (t1 == 0ull) return;
    unsigned long long old = atomicMax(&top[0], t1);
    atomicMax(&top[1], (t1 > old) ? old : t1);
    if (t2) atomicMax(&top[1], t2);
}

// Called by every thread of the block (inactive threads pass valid = false).
// dsq must be >= 0 and finite when valid.
__device__ __forceinline__ void check_accumulate(const DevCtx& c, uint32_t sys_id, bool valid,
                                                 double dsq) {
    __shared__ unsigned long long s1[BLOCK / 32], s2[BLOCK / 32];
    __shared__ uint32_t ssys[BLOCK / 32];
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // dsq >= 0 (a sum of squares) when valid: its bit pattern orders like its
    // value, and +0 is the pattern 0
    unsigned long long v1 = valid ? (unsigned long long)__double_as_longlong(dsq) : 0ull;
    unsigned long long v2 = 0ull;
    uint32_t sid = valid ? sys_id : 0xFFFFFFFFu;
    // warp-level: lanes that hold no value adopt the warp's first valid system
    unsigned vmask = __ballot_sync(0xFFFFFFFFu, valid);
    uint32_t wsys = 0xFFFFFFFFu;
    if (vmask) wsys = __shfl_sync(0xFFFFFFFFu, sid, __ffs(vmask) - 1);
    bool same = __all_sync(0xFFFFFFFFu, !valid || sid == wsys);
    __syncthreads();
    if (same) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            unsigned long long o1 = __shfl_down_sync(0xFFFFFFFFu, v1, off);
            unsigned long long o2 = __shfl_down_sync(0xFFFFFFFFu, v2, off);
            top2_merge(v1, v2, o1, o2);
        }
        if (lane == 0) {
            s1[warp] = v1;
            s2[warp] = v2;
            ssys[warp] = wsys;
        }
    } else {
        if (valid) top2_push(&c.top[2 * (size_t)sid], v1, 0ull);
        if (lane == 0) {
            s1[warp] = 0ull;
            s2[warp] = 0ull;
            ssys[warp] = 0xFFFFFFFFu;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // merge runs of warps that share a system, one push per run
        uint32_t cur = 0xFFFFFFFFu;
        unsigned long long a1 = 0ull, a2 = 0ull;
        for (int w = 0; w < BLOCK / 32; w++) {
            if (ssys[w] == 0xFFFFFFFFu) continue;
            if (ssys[w] != cur) {
                if (cur != 0xFFFFFFFFu) top2_push(&c.top[2 * (size_t)cur], a1, a2);
                cur = ssys[w];
                a1 = s1[w];
                a2 = s2[w];
            } else {
                top2_merge(a1, a2, s1[w], s2[w]);
            }
        }
        if (cur != 0xFFFFFFFFu) top2_push(&c.top[2 * (size_t)cur], a1, a2);
    }
}

// Thread 0 of a block: whether the block is the last of its grid to arrive at
// `counter`.  The block's writes before its last barrier are seen by the last
// block (the fence is cumulative over the barrier; read them through L2:
// __ldcg, atomics), and the counter is left at 0 for the next launch.
__device__ __forceinline__ bool arrive_last(uint32_t* counter, uint32_t blocks) {
    __threadfence();
    if (atomicAdd(counter, 1u) + 1u != blocks) return false;
    atomicExch(counter, 0u);
    __threadfence();
    return true;
}

// the same, asked by every thread of the block
__device__ __forceinline__ bool last_block(uint32_t* counter, uint32_t blocks) {
    __shared__ uint32_t last;
    __syncthreads();
    if (threadIdx.x == 0) last = arrive_last(counter, blocks) ? 1u : 0u;
    __syncthreads();
    return last != 0u;
}

// Arm: decide, per system, whether a rebuild is due, from the forced requests
// and the two largest displacements; counts the build and clears what it
// consumed, and sets the conditional node's value.  Executed by the first
// `threads` threads of a block (32: one warp, no block barrier; else all).
__device__ __forceinline__ void arm_systems(const DevCtx& c, uint32_t threads, int count_step, int use_cond,
                                            cudaGraphConditionalHandle handle) {
    int any = 0;
    for (uint32_t s = threadIdx.x; s < c.nsys; s += threads) {
        if (count_step && !c.active[s]) {
            // frozen system: no rebuild in time steps; its pending test
            // (displacements, forced rebuild) waits until it is stepped again
            c.flag[s] = 0u;
            continue;
        }
        const ulonglong2 top = __ldcg(reinterpret_cast<const ulonglong2*>(c.top) + s);
        const double t1 = __longlong_as_double((long long)top.x), t2 = __longlong_as_double((long long)top.y);
        // reference: bigdist + biggestdist >= skin, evaluated only once some atom moved
        bool rb = c.force_rb[s] != 0u;
        if (!rb && t1 > 0.0) rb = __dadd_rn(__dsqrt_rn(t2), __dsqrt_rn(t1)) >= c.sys[s].skin;
        c.flag[s] = rb ? 1u : 0u;
        if (rb) {
            c.which[s] += 1u;
            c.force_rb[s] = 0u;
        }
        reinterpret_cast<ulonglong2*>(c.top)[s] = make_ulonglong2(0ull, 0ull);
        any |= rb ? 1 : 0;
    }
    if (threads == 32u) any = __any_sync(0xFFFFFFFFu, any);
    else any = __syncthreads_or(any);
    if (threadIdx.x == 0) {
        *c.any_flag = (uint32_t)(any != 0);
        if (any) *c.chains += 1u;
        if (count_step) c.params->step += 1ull;
        if (use_cond) cudaGraphSetConditional(handle, any ? 1u : 0u);
    }
}

// Arm by the last block of a grid (after check_accumulate).  Up to 32 systems,
// one warp of each block sees to it and the others leave at once: a block that
// waits as a whole for its arrival costs large grids a sixth of their time.
__device__ __forceinline__ void arm_by_last_block(const DevCtx& c, int count_step, int use_cond,
                                                  cudaGraphConditionalHandle handle) {
    if (c.nsys <= 32u) {
        if (threadIdx.x >= 32u) return;
        bool last = false;
        if (threadIdx.x == 0) last = arrive_last(&c.done[0], gridDim.x);
        if (__any_sync(0xFFFFFFFFu, last)) arm_systems(c, 32u, count_step, use_cond, handle);
    } else if (last_block(&c.done[0], gridDim.x)) {
        arm_systems(c, blockDim.x, count_step, use_cond, handle);
    }
}

// squared displacement |x - lastloc|^2 in the reference's order
// ((dx*dx + dy*dy) + dz*dz); FP64 without contraction (callers compile with
// -fmad=false or use this routine, which uses explicit round-to-nearest ops)
template <int ND>
__device__ __forceinline__ double disp_sq(const typename DVec<ND>::T& x, const typename DVec<ND>::T& l);
template <>
__device__ __forceinline__ double disp_sq<3>(const double4& x, const double4& l) {
    double dx = __dsub_rn(x.x, l.x), dy = __dsub_rn(x.y, l.y), dz = __dsub_rn(x.z, l.z);
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}
template <>
__device__ __forceinline__ double disp_sq<2>(const double2& x, const double2& l) {
    double dx = __dsub_rn(x.x, l.x), dy = __dsub_rn(x.y, l.y);
    return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
}

}  // namespace parm
