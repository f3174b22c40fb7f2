// Ragged ensembles: many independent Roe-Exner grids (each with its own size, state,
// boundary recipes and dt) advanced together, one launch per phase for all members.
//
// The work items of every member (stage tiles; CFL strips x row bands) are numbered
// consecutively, member after member.  A block (stage: one tile) or a warp (CFL) finds
// the member of its item by binary search in the item offsets and copies that member's
// argument block to shared memory, so the per-item body is exactly the single-grid one
// (re_stage_tile / re_cfl_item) reading its arguments from there.
//
// CFL: each item folds its face speeds into the member's maximum (one 64-bit atomicMax
// per warp and item); a one-thread-per-member launch then turns the maxima into the
// members' dts, logs and resets them.  Each member keeps its own dt, as N separate runs of
// the reference's integrator would.
#pragma once
#include "re_cfl.cuh"
#include "re_stage.cuh"

namespace pxb {

template <class T>
struct EnsStageArgs {
    const REStageArgs<T>* args;  // per member
    const int* base;             // item offset of each member, nmembers + 1 entries
    int nmembers;
};

template <class T>
struct EnsCflArgs {
    const CflArgs<T>* args;  // per member (scr, dt_out, dt_log, cfl, dx, floor per member)
    const int* base;
    int nmembers;
    int log_stride;  // members per dt-log row
};

__device__ __forceinline__ int ens_member_of(const int* base, int nm, int item) {
    int lo = 0, hi = nm - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(base + mid) <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Warp-cooperative copy of one argument block into the warp's shared slot.
template <class A>
__device__ __forceinline__ void ens_load_slot(A* slot, const A* src) {
    static_assert(sizeof(A) % 4 == 0, "argument blocks are copied as 32-bit words");
    const unsigned* s = reinterpret_cast<const unsigned*>(src);
    unsigned* d = reinterpret_cast<unsigned*>(slot);
    __syncwarp();
    for (int k = threadIdx.x & 31; k < (int)(sizeof(A) / 4); k += 32) d[k] = __ldg(s + k);
    __syncwarp();
}

// One block per tile of any member.
template <class T, bool MPM, bool HAS_MASK, bool AVG>
__global__ void __launch_bounds__(stage_max_threads(sizeof(T)), stage_min_blocks(sizeof(T)))
    ens_stage_kernel(const EnsStageArgs<T> e) {
    __shared__ REStageArgs<T> slot;
    const int item = blockIdx.x;
    const int m = ens_member_of(e.base, e.nmembers, item);
    {
        static_assert(sizeof(REStageArgs<T>) % 4 == 0, "argument blocks are copied as 32-bit words");
        const unsigned* src = reinterpret_cast<const unsigned*>(e.args + m);
        unsigned* dst = reinterpret_cast<unsigned*>(&slot);
        for (int k = threadIdx.x; k < (int)(sizeof(slot) / 4); k += blockDim.x) dst[k] = __ldg(src + k);
        __syncthreads();
    }
    const int tile = item - __ldg(e.base + m);
    bool bad = false;
    if (stage_tile_interior(slot, tile)) re_stage_tile<T, MPM, HAS_MASK, AVG, false, true>(slot, tile, stage_shared<T>(), bad);
    else re_stage_tile<T, MPM, HAS_MASK, AVG, false, false>(slot, tile, stage_shared<T>(), bad);
    if (bad) atomicOr(slot.err, 1);
}

// One narrow item per warp (members are small: wide items of 32 rows took about 120 us where
// these take 28 for 3.5 M cells in 24 members; for two members of 2048^2, float32 at rest, they
// take 49 of a step's 420 us).
template <class T, bool HAS_MASK>
__global__ void __launch_bounds__(256, cfl_min_blocks(sizeof(T))) ens_cfl_kernel(const EnsCflArgs<T> e) {
    __shared__ CflArgs<T> slot[8];
    const int w = threadIdx.x >> 5;
    const int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (item >= __ldg(e.base + e.nmembers)) return;  // whole warps
    const int m = ens_member_of(e.base, e.nmembers, item);
    ens_load_slot(&slot[w], e.args + m);
    unsigned long long best = 0ull;
    re_cfl_item<T, HAS_MASK>(slot[w], item - __ldg(e.base + m), best);
    best = warp_max_bits(best);
    if ((threadIdx.x & 31) == 0 && best != 0ull) atomicMax(&slot[w].scr->maxbits, best);
}

// dt of every member from its maximum face speed (as the last block of re_cfl_kernel).
template <class T>
__global__ void ens_cfl_finalize_kernel(const EnsCflArgs<T> e) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= e.nmembers) return;
    const CflArgs<T>& a = e.args[m];
    CflScratch* scr = a.scr;
    const T smax = bits_speed(scr->maxbits, T(0));
    T dt = a.cfl * (a.dx / smax);
    if (a.floor_dt > T(0)) dt = clamp_lo(dt, a.floor_dt);
    *a.dt_out = dt;
    if (a.dt_log) a.dt_log[(long long)scr->step * e.log_stride + m] = dt;
    scr->step += 1;
    if (!d_isfinite(dt)) scr->err |= 2;
    scr->maxbits = 0ull;
}

}  // namespace pxb
