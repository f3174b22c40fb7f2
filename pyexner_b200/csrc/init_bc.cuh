// Set-up kernels: the pointwise part of init_fn_roeexner (n_b and G,
// PyExner src/PyExner/solvers/roe_exner_solver.py:58-78) and the exact, handler-by-handler
// boundary application of BoundaryManager.apply (src/PyExner/domain/boundary_registry.py:183-187).
//
// The generic application runs each handler as a gather of all donor values into a
// scratch buffer followed by a scatter into the boundary cells, which is the jax
// semantics of `state.h.at[by, bx].set(state.h[iy, ix])` (reads before writes within a
// handler, later handlers overwrite earlier ones).  It serves the set-up and the general
// stage path; the fused stage kernel uses the ring recipes resolved from the same handlers.
#pragma once
#include <cooperative_groups.h>

#include "pxb_device.cuh"

namespace pxb {

template <class T>
struct InitArgs {
    int ny, nx;
    long long pitch;
    const T *h, *hu, *hv, *zb, *n;
    T *nb, *G;
    const uint8_t* nodata;
    int mpm;
    SedTable<T> sed;
};

template <class T>
__global__ void __launch_bounds__(256) re_init_kernel(const InitArgs<T> a) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (r >= a.ny || c >= a.nx) return;
    const long long i = (long long)r * a.pitch + c;
    const bool m0 = a.nodata ? (a.nodata[i] != 0) : false;
    if (a.mpm) {
        // compute_n (roe_exner.py:64-73)
        a.nb[i] = a.zb[i] > T(SED_TOL) ? a.sed.n_p_mix : a.n[i];
        a.G[i] = mpm_grass(a.h[i], a.hu[i], a.hv[i], m0, a.sed);
    } else {
        a.nb[i] = a.n[i];
        a.G[i] = const_grass(a.h[i], a.G[i], m0);
    }
}

// Field slots of the generic handler kernels (a null slot is skipped).
//   Roe-Exner: 0 h, 1 hu, 2 hv, 3 z_b, 4 n, 5 G
//   Roe:       0 h, 1 hu, 2 hv, 3 z,   4 n, 5 (unused)
template <class T>
struct BcHandler {
    const long long* cells;
    const long long* donors;
    int count;
    int kind;
    T nx, ny;
    T c0, c1;             // constant momenta (ConstantInflux, ConstantOutflux, ZeroMomentum; NaN = keep)
    T q, vx, vy;          // ConstantOutflux: discharge and direction (float32 values)
    float neg_alpha, zb0;  // Berthon / NormalFlowDepth: z_b = fl32(fl32(neg_alpha * fl32(t)) + zb0)
    T hb;                 // NormalFlowDepth: depth q/u
    int off;              // its first value of each slot in tmp
    int level;            // reads a value that a handler since the last level writes: a new level
    int barrier;          // writes a value that a handler since the last barrier writes
};

template <class T>
struct BcFields {
    T* f[6];
    const double* tptr;   // simulation time on the device, or null: use tval
    double tval;
    T* tmp;               // 6 * total values (handlers in two launches)
    int total;            // boundary cells of all handlers
};

template <class T>
struct BcArgs {  // one handler
    BcFields<T> f;
    BcHandler<T> h;
};

// Handlers one launch applies, threads of a block and blocks of its cluster: a level has at
// most as many warps' worth of boundary cells (chunks of 32 of a handler).
constexpr int BC_SET_MAX = 16, BC_SET_THREADS = 512, BC_SET_BLOCKS = 8;
constexpr int BC_SET_CHUNKS = BC_SET_THREADS / 32 * BC_SET_BLOCKS;
template <class T>
struct BcSet {
    BcFields<T> f;
    int n;
    BcHandler<T> h[BC_SET_MAX];
};

// Depth of a ConstantOutflux cell: five Newton steps on the outgoing Riemann invariant
// of the donor, q/h + 2 sqrt(g h) = un + 2 sqrt(g h_i) (roeexner_constantoutflux.py:29-58).
template <class T>
__device__ __forceinline__ T outflux_depth(T h, T hu, T hv, T q, T vx, T vy) {
    const T G = T(9.81), TINY = T(1e-8);
    const T h_i = nan_max(h, TINY);
    const T u_i = hu / h_i, v_i = hv / h_i;
    const T un_i = u_i * vx + v_i * vy;
    const T rp = un_i + T(2) * d_sqrt(G * h_i);
    T hb = h_i;
    for (int it = 0; it < 5; ++it) {
        hb = nan_max(hb, TINY);
        const T c = d_sqrt(G * hb);
        const T f = q / hb + T(2) * c - rp;
        const T df = -q / (hb * hb) + G / nan_max(c, TINY);
        hb = nan_max(hb - f / df, TINY);
    }
    return hb;
}

// z_b of the Berthon analytic solution at time t, in float32 like the reference's
// float32 values (roeexner_berthon.py:49-52): -alpha * t + zb0.
__device__ __forceinline__ float berthon_zb(float neg_alpha, float zb0, double t) {
    return __fadd_rn(__fmul_rn(neg_alpha, __double2float_rn(t)), zb0);
}

// A value past the L1 (another SM may have written it in this launch).
template <class T>
__device__ __forceinline__ T bc_load(const T* p) {
    if constexpr (sizeof(T) == 16) {  // a dual number
        const double2 t = __ldcg(reinterpret_cast<const double2*>(p));
        T x;
        x.v = t.x;
        x.d = t.y;
        return x;
    } else {
        return __ldcg(p);
    }
}

// Values t[slot] of a boundary cell of a handler from its donor d.
template <class T>
__device__ __forceinline__ void bc_values(const BcFields<T>& F, const BcHandler<T>& h, const long long d, T (&t)[6]) {
    auto ld = [&](int slot) { return F.f[slot] ? bc_load(F.f[slot] + d) : T(0); };  // null slots read as 0
    switch (h.kind) {
        case PXB_BC_RE_REFLECTIVE: {  // roeexner_reflective.py:17-63
            const T hu = ld(1), hv = ld(2);
            const T mom_n = hu * h.nx + hv * h.ny;
            const T mom_t = -hu * h.ny + hv * h.nx;
            const T mom_r = -mom_n;
            t[0] = ld(0);
            t[1] = mom_r * h.nx - mom_t * h.ny;
            t[2] = mom_r * h.ny + mom_t * h.nx;
            t[3] = ld(3);
            t[4] = ld(4);
            t[5] = ld(5);
            break;
        }
        case PXB_BC_RE_TRANSMISSIVE:  // roeexner_transmissive.py:17-31
            t[0] = ld(0);
            t[1] = ld(1);
            t[2] = ld(2);
            break;
        case PXB_BC_RE_TRANSMISSIVEBED:  // roeexner_transmissivebed.py:17-27
            t[3] = ld(3);
            break;
        case PXB_BC_RE_CONSTANTINFLUX:  // roeexner_constantinflux.py:18-48
            t[1] = h.c0;
            t[2] = h.c1;
            break;
        case PXB_BC_ROE_REFLECTIVE:  // roe_reflective.py:18-44
            t[0] = ld(0);
            t[3] = ld(3);
            t[4] = ld(4);
            t[1] = ld(1) * (T(1) - T(2) * h.nx * h.nx);
            t[2] = ld(2) * (T(1) - T(2) * h.ny * h.ny);
            break;
        case PXB_BC_ROE_TRANSMISSIVE:  // roe_transmissive.py:17-43
            t[0] = ld(0);
            t[1] = ld(1);
            t[2] = ld(2);
            t[3] = ld(3);
            t[4] = ld(4);
            break;
        case PXB_BC_RE_CONSTANTOUTFLUX:  // roeexner_constantoutflux.py:18-73
            t[0] = outflux_depth(ld(0), ld(1), ld(2), h.q, h.vx, h.vy);
            t[1] = h.c0;
            t[2] = h.c1;
            break;
        case PXB_BC_RE_BERTHON:  // roeexner_berthon.py:19-56
            t[3] = T(berthon_zb(h.neg_alpha, h.zb0, F.tptr ? *F.tptr : F.tval));
            break;
        case PXB_BC_RE_NORMALFLOWDEPTH:  // roeexner_normalflowdepth.py:19-51
            t[0] = h.hb;
            t[1] = ld(1);
            t[2] = ld(2);
            t[3] = T(berthon_zb(h.neg_alpha, h.zb0, F.tptr ? *F.tptr : F.tval));
            break;
        case PXB_BC_RE_STEEPFALL:  // roeexner_steepfall.py:17-26
            t[3] = ld(3) - T(1);
            break;
        case PXB_BC_RE_ZEROMOMENTUM:  // roeexner_zeromomentum.py:16-31; the donor is the cell
            t[1] = (h.c0 != h.c0) ? ld(1) : h.c0;
            t[2] = (h.c1 != h.c1) ? ld(2) : h.c1;
            break;
        default:
            break;
    }
}

__host__ __device__ inline unsigned bc_field_mask(int kind) {
    switch (kind) {
        case PXB_BC_RE_REFLECTIVE: return 0x3f;
        case PXB_BC_RE_TRANSMISSIVE: return 0x07;
        case PXB_BC_RE_TRANSMISSIVEBED: return 0x08;
        case PXB_BC_RE_CONSTANTINFLUX: return 0x06;
        case PXB_BC_ROE_REFLECTIVE: return 0x1f;
        case PXB_BC_ROE_TRANSMISSIVE: return 0x1f;
        case PXB_BC_RE_CONSTANTOUTFLUX: return 0x07;
        case PXB_BC_RE_BERTHON: return 0x08;
        case PXB_BC_RE_NORMALFLOWDEPTH: return 0x0f;
        case PXB_BC_RE_STEEPFALL: return 0x08;
        case PXB_BC_RE_ZEROMOMENTUM: return 0x06;
        default: return 0;
    }
}

// Fields a handler reads at its donors (the cells themselves for ZeroMomentum).
__host__ __device__ inline unsigned bc_read_mask(int kind) {
    switch (kind) {
        case PXB_BC_RE_CONSTANTINFLUX:
        case PXB_BC_RE_BERTHON: return 0;
        case PXB_BC_RE_NORMALFLOWDEPTH: return 0x06;
        default: return bc_field_mask(kind);
    }
}

template <class T>
__device__ __forceinline__ void bc_store(const BcFields<T>& F, const BcHandler<T>& h, const long long b, const T (&t)[6]) {
    const unsigned fm = bc_field_mask(h.kind);
#pragma unroll
    for (int s = 0; s < 6; ++s)
        if (((fm >> s) & 1u) && F.f[s]) F.f[s][b] = t[s];
}

// One handler in two launches (layouts above BC_SET_CELLS): gather into the temporary,
// scatter into the cells.
template <class T>
__global__ void bc_gather_kernel(const BcArgs<T> a) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.h.count) return;
    T t[6] = {};
    bc_values(a.f, a.h, a.h.donors[k], t);
#pragma unroll
    for (int s = 0; s < 6; ++s) a.f.tmp[(size_t)s * a.f.total + a.h.off + k] = t[s];
}

template <class T>
__global__ void bc_scatter_kernel(const BcArgs<T> a) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.h.count) return;
    T t[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) t[s] = a.f.tmp[(size_t)s * a.f.total + a.h.off + k];
    bc_store(a.f, a.h, a.h.cells[k], t);
}

// All handlers by one cluster of blocks, one boundary cell of a level per thread.  Handlers
// that read nothing the ones before them write form a level: all of a level's values are
// read before any is written, and within the level a later handler's values are written
// after those they overwrite (a barrier only where two write the same value).  The same
// results as one handler after the other.  A warp takes 32 cells of one handler; the next
// level's indices are read before the barriers of this one.  Bound by the chain of value,
// barrier and store latencies of each level.  Two launches per handler took 4.6 us, 37 us
// for 8 handlers of 2500 cells; one block with the values in global scratch 17.3 us, this 6.9
// (dual numbers 15.3 and 8.0).
template <class T>
__global__ void __launch_bounds__(BC_SET_THREADS) bc_set_kernel(const __grid_constant__ BcSet<T> a) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31;
    const int warp = (int)cluster.block_rank() * (blockDim.x >> 5) + (threadIdx.x >> 5);
    // this thread's handler (-1: none), cell and donor among the handlers h0 .. h1-1
    struct Item { int q; long long cell, donor; };
    auto locate = [&](int h0, int h1) {
        Item it{-1, 0, 0};
        int chunk = warp;
        for (int q = h0; q < h1; ++q) {
            const int chunks = (a.h[q].count + 31) >> 5;
            if (chunk < chunks) {
                const int k = 32 * chunk + lane;
                if (k < a.h[q].count) it = Item{q, a.h[q].cells[k], a.h[q].donors[k]};
                break;
            }
            chunk -= chunks;
        }
        return it;
    };
    auto level_end = [&](int h0) {
        int h1 = h0 + 1;
        while (h1 < a.n && !a.h[h1].level) ++h1;
        return h1;
    };
    int h0 = 0, h1 = level_end(0);
    Item it = locate(h0, h1);
    while (h0 < a.n) {
        T t[6] = {};
        if (it.q >= 0) bc_values(a.f, a.h[it.q], it.donor, t);
        const int n1 = h1 < a.n ? level_end(h1) : h1;
        const Item next = h1 < a.n ? locate(h1, n1) : Item{-1, 0, 0};
        cluster.sync();
        for (int q = h0; q < h1;) {
            int e = q + 1;
            while (e < h1 && !a.h[e].barrier) ++e;
            if (it.q >= q && it.q < e) bc_store(a.f, a.h[it.q], it.cell, t);
            q = e;
            if (q < h1 || h1 < a.n) {  // (nothing follows the last handlers' stores)
                __threadfence();
                cluster.sync();
            }
        }
        it = next;
        h0 = h1;
        h1 = n1;
    }
}

}  // namespace pxb
