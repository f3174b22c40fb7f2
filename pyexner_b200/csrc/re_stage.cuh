// Fused Roe-Exner stage kernel (one launch per Runge-Kutta stage).
//
// Replaces step_fn_roeexner (PyExner src/PyExner/solvers/roe_exner_solver.py:80-116) on
// one rank: hydro update (roe_exner.py:535-612) -> momentum corrections (:14-62) ->
// boundary handlers -> grass factor (:85-140) -> Exner update (:665-717) -> boundary
// handlers, and for the second SSPRK2 stage the 0.5/0.5 combination (SSPRK2.py:40).
//
// Layout of the work: a block computes one tile, a strip of 30 wx - 4 owned columns by a
// band of owned rows, in two phases with the updated h, hu, hv of the tile (two halo rows
// and columns on each side) in shared memory between them:
//   1  hydro faces and update: its warps stand wx side by side and wy on top of one
//      another; a warp holds 32 columns, of which the inner 30 get both of their x-faces
//      from shuffles (side-by-side warps overlap by two columns), and marches down its
//      share of the rows with the north face's fluctuation in registers
//   C  momentum corrections, only where some cell of the tile is dry (or masked), and the
//      first boundary application, only in tiles with ring cells, in shared memory
//   2  grass factor, Exner cells, faces and z_b update, the same march, then the stores;
//      ring cells are finished last, from their donors' values in shared memory (second
//      boundary application)
// A face between two warps' row shares is evaluated by both; every other face of a tile
// is evaluated once.  Warp votes skip work whose result is known for the whole warp: the
// entropy fix and the wave split where every face is subcritical, the activity masks where
// every cell is wet, the grass factor and the Exner update where no cell near the warp's
// carries sediment.
//
// Bound by instruction issue (79 and 77 % of issue slots in the two float32 stages at 2048^2,
// DRAM at 18 and 28 %).  The tile replaced a warp that marched down a band with all phases in one
// register pipeline: that needed 118 registers (16 warps per SM, 74 % of issue slots),
// moved 35 values a row between pipeline stages, repeated 1.41 times the cells (32 columns
// for 26) and ran 11 rows before its first store, which set the time of small grids.
// Measured, before -> after, us per SSPRK2 step with the CFL reduction (float32):
// 48^2 51.5 -> 23, 256^2 53.6 -> 26.7, 512^2 60.7 -> 35, 1024^2 105 -> 66, 2048^2 252 ->
// 203, 8192^2 3200 -> 2550; with bedload in every cell 2048^2 328 -> 309.
#pragma once
#include "pxb_device.cuh"

// Threads of the largest block and resident blocks of that size per SM the stage kernels
// are register-limited to.  float32: 2 x 384 threads (80 registers, a few spilled bytes);
// 2 x 512 (64 registers, 56 B of spills) is 5 % slower at 2048^2 and 10 % at 8192^2.
// float64: 2 x 256 (128 registers); 3 x 256 is 5 % slower with bedload everywhere and 25 %
// without, 2 x 384 like it, 4 x 256 (64 registers, 1.2 KB of spills) 30 to 50 % slower.
#ifndef PXB_STAGE_THREADS_F32
#define PXB_STAGE_THREADS_F32 384
#endif
#ifndef PXB_STAGE_BLOCKS_F32
#define PXB_STAGE_BLOCKS_F32 2
#endif
#ifndef PXB_STAGE_THREADS_F64
#define PXB_STAGE_THREADS_F64 256
#endif
#ifndef PXB_STAGE_BLOCKS_F64
#define PXB_STAGE_BLOCKS_F64 2
#endif
// Rows of the averaging stage whose partner values are loaded together, one batch ahead of
// the batch being stored (and the first before the block's barrier): 3 against 2 and 4 is
// 1 to 3 % faster at 8192^2; without the batch ahead the averaging stage took 1410 us there
// instead of 1210.
#ifndef PXB_STAGE_BATCH
#define PXB_STAGE_BATCH 3
#endif

namespace pxb {

constexpr int stage_max_threads(int esize) { return esize == 8 ? PXB_STAGE_THREADS_F64 : PXB_STAGE_THREADS_F32; }
constexpr int stage_min_blocks(int esize) { return esize == 8 ? PXB_STAGE_BLOCKS_F64 : PXB_STAGE_BLOCKS_F32; }

// Columns of a tile with wx warps side by side: all (raw), and owned by an inner strip.
static inline constexpr __host__ __device__ int stage_cols(int wx) { return 30 * wx + 2; }
static inline constexpr __host__ __device__ int stage_owned(int wx) { return 30 * wx - 4; }
// Strips of a grid: the first owns three columns more (no halo to its west), the last up
// to three more; every strip but the first starts where its left neighbour's ends.
static inline __host__ __device__ int stage_strips(int nx, int wx) {
    const int oc = stage_owned(wx);
    return nx > 6 + oc ? (nx - 6 + oc - 1) / oc : 1;
}
// First row of band b: bands differ by at most one row (and have at least two: the host
// asks for at most ny / 2 bands).
static inline __host__ __device__ int stage_band_row(int ny, int nbands, int b) {
    return (int)(((long long)ny * b) / nbands);
}
// Shared memory of a block, in elements: h, hu, hv of srows x cols cells, and for ring
// cells five values per slot (first application: h, hu, hv, then z_b and G) and z_b, G of
// the four outermost rows and columns.
static inline __host__ __device__ size_t stage_smem_elems(int wx, int srows) {
    const size_t pw = stage_cols(wx);
    return 3 * pw * srows + 12 * (pw + srows);
}

template <class T>
struct REStageArgs {
    int ny, nx;
    long long pitch;
    T dx;
    const T *h, *hu, *hv, *zb, *z, *nb, *G;  // stage input (G read in constant-G mode)
    const uint8_t* nodata;                    // mask[0] or null
    T *oh, *ohu, *ohv, *ozb, *oG;            // stage output (oG may be null)
    const T *ah, *ahu, *ahv, *azb, *aG;      // SSPRK2 partner u^n (AVG)
    const T* dt;
    const pxb_ring_recipe* ring;              // null when there are no handlers
    SedTable<T> sed;
    int wx, srows, nstrips, nbands;  // tiles: warps side by side, shared rows, strips, bands
    int* err;
    // Volume budget (null: off): per tile, the outflow through the outer boundary of the
    // physical cells (rows and columns 1 .. n-2) of water (sum of the mass fluxes of the
    // boundary faces) and of sediment (Exner fluxes), in the state's flux units; tile k
    // writes bud[2k], bud[2k+1] on every launch.
    double* bud;
};

template <class T>
__device__ __forceinline__ HCell<T> shfl_down_hcell(const HCell<T>& p) {
    HCell<T> q;
    q.h = __shfl_down_sync(FULL, p.h, 1);
    q.u = __shfl_down_sync(FULL, p.u, 1);
    q.v = __shfl_down_sync(FULL, p.v, 1);
    q.sq = __shfl_down_sync(FULL, p.sq, 1);
    q.c = __shfl_down_sync(FULL, p.c, 1);
    q.zt = __shfl_down_sync(FULL, p.zt, 1);
    q.nb = __shfl_down_sync(FULL, p.nb, 1);
    return q;
}

template <class T>
__device__ __forceinline__ ECell<T> shfl_down_ecell(const ECell<T>& p) {
    ECell<T> q;
    q.h = __shfl_down_sync(FULL, p.h, 1);
    q.zb = __shfl_down_sync(FULL, p.zb, 1);
    q.zbe = __shfl_down_sync(FULL, p.zbe, 1);
    q.sq = __shfl_down_sync(FULL, p.sq, 1);
    q.u = __shfl_down_sync(FULL, p.u, 1);
    q.v = __shfl_down_sync(FULL, p.v, 1);
    q.um = __shfl_down_sync(FULL, p.um, 1);
    q.G = __shfl_down_sync(FULL, p.G, 1);
    return q;
}

// One row of this lane's column as read from HBM.
template <class T>
struct RawCell {
    T h, hu, hv, zb, z, nb;
    bool m;
};

// The SSPRK2 partner's values of one cell.
template <class T>
struct Partner {
    T h, hu, hv, zb, G;
};

// One tile.  INTERIOR: the instantiation for tiles away from the grid's boundary (inner
// strips of inner bands): every column lies inside the grid and no cell whose Exner
// update the tile needs is a ring cell, so it carries neither column tests nor boundary
// code.  The results do not depend on the tiling.
template <class T, bool MPM, bool HAS_MASK, bool AVG, bool BUD, bool INTERIOR>
__device__ __forceinline__ void re_stage_tile(const REStageArgs<T>& a, const int tile, T* const S, bool& bad) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wx = a.wx, wy = (int)(blockDim.x >> 5) / wx;
    const int iy = warp / wx, ix = warp - iy * wx;
    const int ny = a.ny, nx = a.nx;
    const unsigned upitch = (unsigned)a.pitch;  // planes are < 2^31 elements (checked at plan creation)
    const T dt = *a.dt;
    const T dx = a.dx;
    const T dtdx = dt / dx;  // float path only
    const T DRY = T(DRY_TOL);
    const int band = tile / a.nstrips, strip = tile - band * a.nstrips;
    const bool first_strip = strip == 0, last_strip = strip == a.nstrips - 1;
    const int pw = stage_cols(wx), sr = a.srows;
    const int cstart = strip * stage_owned(wx);  // column of index 0
    const int idx = 30 * ix + lane, c = cstart + idx;
    const bool colok = INTERIOR || c < nx;
    const bool has_e = lane < 31 && (INTERIOR || c + 1 < nx);
    // owned columns by index, and the lane of the column's one owner
    const int lo = first_strip ? 0 : 3, hi = last_strip ? nx - 1 - cstart : pw - 4;
    const bool lane_in = (lane >= 1 && lane <= 30) || (idx == 0) || (idx == pw - 1);
    const bool out_col = lane_in && idx >= lo && idx <= hi;
    const bool near_col = lane_in && idx >= lo - 1 && idx <= hi + 1 && colok;  // owned or next to one
    const int R0 = stage_band_row(ny, a.nbands, band), R1 = stage_band_row(ny, a.nbands, band + 1);
    const int H0 = max(0, R0 - 2), H1 = min(ny, R1 + 2);  // rows of the hydro update
    const int K0 = max(0, R0 - 1), K1 = min(ny, R1 + 1);  // rows of the Exner cells
    T* const Sh = S;
    T* const Su = S + (size_t)pw * sr;
    T* const Sv = S + 2 * (size_t)pw * sr;
    auto sidx = [&](int r, int k) __attribute__((always_inline)) { return (r - (R0 - 2)) * pw + k; };
    // Budget: a face counts once, in the tile that owns its row (x-faces; y-faces (r-1|r)
    // by row r) and the lane that owns the column.  The outflow of a face with left cell I
    // (west / north side) is F = h_I u_n,I + upwM_0, the flux whose differences the
    // fluctuations of roe_exner.py:597-606 telescope to; F leaves the physical cells
    // through the east / south boundary and enters them through the west / north one.
    // Exner: the upwind face flux of roe_exner.py:708-715.
    double budh = 0.0, budz = 0.0;

    // ================= phase 1: hydro faces and update of rows H0 .. H1-1
    // One writer per cell: the column's owner lane, where both of its x-faces lie in the warp.
    // Neighbouring warps overlap by two columns, so the grid's last column may also be lane 0
    // of a warp, which lacks its west face.  The outermost index columns miss a face unless the
    // grid ends there: they stay zero, as do the columns beyond the grid.
    const bool inner_lane = lane >= 1 && lane <= 30;
    const bool whole = INTERIOR ? inner_lane : lane_in && colok && (inner_lane || c == 0 || c == nx - 1);
    bool dry = false;
    {
        if (lane_in && !whole)
            for (int r = H0 + iy; r < H1; r += wy) Sh[sidx(r, idx)] = Su[sidx(r, idx)] = Sv[sidx(r, idx)] = T(0);
        const int n = H1 - H0;
        const int q0 = H0 + n * iy / wy, q1 = H0 + n * (iy + 1) / wy;
        auto load = [&](int r) __attribute__((always_inline)) {
            RawCell<T> x;
            if (colok && r >= 0 && r < ny) {
                const unsigned i = (unsigned)r * upitch + (unsigned)c;
                x.h = __ldg(a.h + i);
                x.hu = __ldg(a.hu + i);
                x.hv = __ldg(a.hv + i);
                x.zb = __ldg(a.zb + i);
                x.z = __ldg(a.z + i);
                x.nb = __ldg(a.nb + i);
                x.m = HAS_MASK ? __ldg(a.nodata + i) != 0 : false;
            } else {
                x.h = x.hu = x.hv = x.zb = x.z = x.nb = T(0);
                x.m = false;
            }
            return x;
        };
        if (q0 < q1) {
            int r = max(q0 - 1, 0);  // the row above the share gives its first north face
            RawCell<T> cur = load(r), nxt = load(r + 1);
            HCell<T> p = make_hcell(cur.h, cur.hu, cur.hv, cur.zb, cur.z, cur.nb);
            T nP[3] = {T(0), T(0), T(0)};
            for (; r < q1; ++r) {
                const HCell<T> ps = make_hcell(nxt.h, nxt.hu, nxt.hv, nxt.zb, nxt.z, nxt.nb);
                const T h_r = cur.h, hu_r = cur.hu, hv_r = cur.hv;
                const bool m_r = cur.m;
                cur = nxt;
                if (r + 2 <= q1) nxt = load(r + 2);  // in flight during this row's faces
                // pr.h = max(h, DRY_TOL) > DRY_TOL exactly when h > DRY_TOL (false for NaN).
                // Where every cell of row r is wet (and, with a mask plane, no cell of rows r
                // and r+1 is nodata), all of its x-faces and south faces are active and need no
                // masks (inner tiles; the two outer lanes' missing faces enter no cell that is
                // kept).
                const bool wet = p.h > DRY;
                const bool allwet = INTERIOR && __all_sync(FULL, wet && !(HAS_MASK && (m_r || cur.m)));
                T yP[3] = {T(0), T(0), T(0)}, yM[3] = {T(0), T(0), T(0)};
                if (r + 1 < ny) {
                    roe_exner_face<T, true, true>(p, ps, dx, yP, yM);
                    if (!allwet) {
                        const bool act = colok && (wet || ps.h > DRY) && !(HAS_MASK && (m_r || cur.m));
#pragma unroll
                        for (int m = 0; m < 3; ++m) {
                            yP[m] = act ? yP[m] : T(0);
                            yM[m] = act ? yM[m] : T(0);
                        }
                        if constexpr (BUD && !INTERIOR) {
                            const int rs = r + 1;  // the face (r | r+1) counts with row r+1
                            if (act && out_col && (rs == 1 || rs == ny - 1) && rs >= R0 && rs < R1 && rs >= q0 && rs < q1 &&
                                c >= 1 && c <= nx - 2) {
                                // y-faces have the normal (0, -1): u_n = -v
                                const double F = -(double)mul_rn(p.h, p.v) + (double)yM[0];
                                budh += rs == 1 ? -F : F;
                            }
                        }
                    }
                }
                if (r >= q0) {
                    const HCell<T> pe = shfl_down_hcell(p);
                    const bool me = HAS_MASK ? (__shfl_down_sync(FULL, (int)m_r, 1) != 0) : false;
                    T P[3], M[3];
                    roe_exner_face<T, false, true>(p, pe, dx, P, M);
                    if (!allwet) {
                        const bool act = has_e && (wet || pe.h > DRY) && !(HAS_MASK && (m_r || me));
#pragma unroll
                        for (int m = 0; m < 3; ++m) {
                            P[m] = act ? P[m] : T(0);
                            M[m] = act ? M[m] : T(0);
                        }
                        if constexpr (BUD && !INTERIOR) {
                            if (act && out_col && r >= R0 && r < R1 && r >= 1 && r <= ny - 2 && (c == 0 || c == nx - 2)) {
                                const double F = (double)mul_rn(p.h, p.u) + (double)M[0];
                                budh += c == 0 ? -F : F;
                            }
                        }
                    }
                    // scatter order of roe_exner.py:597-602: east upwM, west upwP, south upwM,
                    // north upwP (lane 0 has no west face in the warp; inactive faces add zeros)
                    T f[3];
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const T w = __shfl_up_sync(FULL, P[m], 1);
                        f[m] = (T(0) + M[m]) + ((INTERIOR || lane > 0) ? w : T(0));
                        f[m] = f[m] + yM[m];
                        f[m] = f[m] + nP[m];
                    }
                    T h1, u1, v1;
                    if constexpr (is_f32<T>()) {
                        h1 = h_r - dtdx * f[0];
                        u1 = hu_r - dtdx * f[1];
                        v1 = hv_r - dtdx * f[2];
                    } else {
                        h1 = h_r - dt * f[0] / dx;
                        u1 = hu_r - dt * f[1] / dx;
                        v1 = hv_r - dt * f[2] / dx;
                    }
                    if (whole) {
                        const int k = sidx(r, idx);
                        Sh[k] = h1;
                        Su[k] = u1;
                        Sv[k] = v1;
                        dry = dry || !(h1 > DRY) || (HAS_MASK && m_r);
                    }
                }
                nP[0] = yP[0];
                nP[1] = yP[1];
                nP[2] = yP[2];
                p = ps;
            }
        }
    }

    // The averaging stage's partner values of this lane's cells of the first rows it will
    // store, in flight across the barrier and the tests that follow.
    constexpr int U = PXB_STAGE_BATCH;
    const int p0 = R0 + (R1 - R0) * iy / wy, p1 = R0 + (R1 - R0) * (iy + 1) / wy;  // rows of phase 2
    auto partner = [&](int p) __attribute__((always_inline)) {
        Partner<T> q{};
        if (AVG && out_col && p < p1) {
            const unsigned i = (unsigned)p * upitch + (unsigned)c;
            q.h = a.ah[i];
            q.hu = a.ahu[i];
            q.hv = a.ahv[i];
            q.zb = a.azb[i];
            if (a.oG) q.G = a.aG[i];
        }
        return q;
    };
    Partner<T> qn[U];
#pragma unroll
    for (int u = 0; u < U; ++u) qn[u] = partner(p0 + u);

    // ================= momentum corrections (roe_exner.py:14-62) of rows K0 .. K1-1
    // Where every cell of the tile is wet and none is nodata no correction applies.  A NaN
    // depth fails `h > DRY`, as it fails `active`.
    dry = __syncthreads_or(dry) != 0;
    if (dry) {
        const int n = K1 - K0;
        const int q0 = K0 + n * iy / wy, q1 = K0 + n * (iy + 1) / wy;
        if (near_col && (INTERIOR || (c >= 1 && c <= nx - 2))) {
            for (int r = max(q0, 1); r < min(q1, ny - 1); ++r) {
                const unsigned i = (unsigned)r * upitch + (unsigned)c;
                const int k = sidx(r, idx);
                const T hc = Sh[k], hE = Sh[k + 1], hW = Sh[k - 1], hN = Sh[k - pw], hS = Sh[k + pw];
                auto zt = [&](unsigned j) __attribute__((always_inline)) { return __ldg(a.z + j) + __ldg(a.zb + j); };
                auto nod = [&](unsigned j) __attribute__((always_inline)) { return HAS_MASK && __ldg(a.nodata + j) != 0; };
                const T eta = hc + zt(i);
                const bool stop_u = ((hE < DRY) && (eta < zt(i + 1))) || ((hW < DRY) && (eta < zt(i - 1))) || nod(i + 1) || nod(i - 1);
                const bool stop_v = ((hN < DRY) && (eta < zt(i - upitch))) || ((hS < DRY) && (eta < zt(i + upitch))) ||
                                    nod(i - upitch) || nod(i + upitch);
                const bool active = (hc > DRY) && !nod(i);
                if (!active || stop_u) Su[k] = T(0);
                if (!active || stop_v) Sv[k] = T(0);
            }
        }
        __syncthreads();
    }

    // ================= first boundary application, on the ring cells of rows K0 .. K1-1
    // Ring slots of the tile: row 0 by index, row ny-1 by index, column 0 by row, column
    // nx-1 by row (the corners belong to the rows).  The recipes map values from before the
    // application, so the new values are gathered before any is written.
    const bool ring_tile = !INTERIOR;
    const int nslots = 2 * (pw + sr);
    T* const slot_v = S + 3 * (size_t)pw * sr;         // gathered h, hu, hv; then rows / columns of z_b, G
    T* const slot_zb = slot_v + 8 * (size_t)(pw + sr);  // z_b and G of the ring cells after the application
    T* const slot_g = slot_zb + nslots;
    auto slot_cell = [&](int k, int& r, int& j) __attribute__((always_inline)) {  // false: not a ring cell of this tile
        bool ok;
        if (k < 2 * pw) {
            r = k < pw ? 0 : ny - 1;
            j = k < pw ? k : k - pw;
            ok = k < pw ? R0 == 0 : R1 == ny;
        } else {
            const int s = k - 2 * pw;
            r = R0 - 2 + (s < sr ? s : s - sr);
            j = s < sr ? -cstart : nx - 1 - cstart;
            ok = r >= max(K0, 1) && r < min(K1, ny - 1) && (s < sr ? first_strip : last_strip);
        }
        return ok && j >= lo - 1 && j <= hi + 1 && cstart + j < nx;
    };
    auto recipe = [&](int r, int j) __attribute__((always_inline)) {
        pxb_ring_recipe rc{};
        if (a.ring) rc = a.ring[ring_slot(r, cstart + j, ny, nx)];
        return rc;
    };
    // h, hu, hv of a ring cell by its recipe from the shared values
    auto apply_hydro = [&](const pxb_ring_recipe& rc, int k0, T& h, T& hu, T& hv) __attribute__((always_inline)) {
        h = (rc.flags & 1u) ? Sh[k0 + rc.h_dy * pw + rc.h_dx] : Sh[k0];
        hu = Su[k0];
        hv = Sv[k0];
        if (rc.flags & 2u) {
            if (rc.flags & 4u) {
                hu = T(rc.m[0]);
                hv = T(rc.m[1]);
            } else {
                const int kd = k0 + rc.m_dy * pw + rc.m_dx;
                const T du = Su[kd], dv = Sv[kd];
                hu = sum2(T(rc.m[0]), du, T(rc.m[1]), dv);
                hv = sum2(T(rc.m[2]), du, T(rc.m[3]), dv);
            }
        }
    };
    if (ring_tile) {
        for (int k = threadIdx.x; k < nslots; k += blockDim.x) {
            int r, j;
            if (!slot_cell(k, r, j)) continue;
            const pxb_ring_recipe rc = recipe(r, j);
            apply_hydro(rc, sidx(r, j), slot_v[k], slot_v[nslots + k], slot_v[2 * nslots + k]);
            const unsigned i = (unsigned)r * upitch + (unsigned)(cstart + j);
            slot_zb[k] = __ldg(a.zb + ((rc.flags & 8u) ? i + (unsigned)((int)rc.zb_dy * (int)upitch + rc.zb_dx) : i));
            if (!MPM) slot_g[k] = __ldg(a.G + ((rc.flags & 16u) ? i + (unsigned)((int)rc.g_dy * (int)upitch + rc.g_dx) : i));
        }
        __syncthreads();
        for (int k = threadIdx.x; k < nslots; k += blockDim.x) {
            int r, j;
            if (!slot_cell(k, r, j)) continue;
            const int s = sidx(r, j);
            Sh[s] = slot_v[k];
            Su[s] = slot_v[nslots + k];
            Sv[s] = slot_v[2 * nslots + k];
        }
        __syncthreads();
    }

    // z_b and G of the four outermost rows (0, 1, ny-2, ny-1) by index and the four
    // outermost columns by row, for the second application
    T* const edge_z = slot_v;
    T* const edge_g = slot_v + 4 * (pw + sr);

    // ================= phase 2: Exner update and stores of rows R0 .. R1-1
    {
        // Final values of a cell of row p: stored, unless it is a ring cell (those are
        // finished last); tiles at the boundary also keep z_b and G of the outermost rows
        // and columns for that.
        auto finish = [&](int p, T oh, T ou, T ov, T zo, T go, const Partner<T>& q) __attribute__((always_inline)) {
            if (!out_col) return;
            if (!INTERIOR) {
                if (p <= 1) { edge_z[p * pw + idx] = zo; edge_g[p * pw + idx] = go; }
                if (p >= ny - 2) {
                    const int w = (4 - (ny - p)) * pw + idx;  // ny-2 -> 2, ny-1 -> 3
                    edge_z[w] = zo;
                    edge_g[w] = go;
                }
                const int w = 4 * pw + p - (R0 - 2);
                if (c <= 1) { edge_z[w + c * sr] = zo; edge_g[w + c * sr] = go; }
                if (c >= nx - 2) {
                    edge_z[w + (4 - (nx - c)) * sr] = zo;
                    edge_g[w + (4 - (nx - c)) * sr] = go;
                }
                if (p == 0 || p == ny - 1 || c == 0 || c == nx - 1) return;
            }
            const unsigned i = (unsigned)p * upitch + (unsigned)c;
            if (AVG) {
                oh = T(0.5) * q.h + T(0.5) * oh;
                ou = T(0.5) * q.hu + T(0.5) * ou;
                ov = T(0.5) * q.hv + T(0.5) * ov;
                zo = T(0.5) * q.zb + T(0.5) * zo;
                go = T(0.5) * q.G + T(0.5) * go;
            }
            a.oh[i] = oh;
            a.ohu[i] = ou;
            a.ohv[i] = ov;
            a.ozb[i] = zo;
            if (a.oG) a.oG[i] = go;
            bad |= !(d_isfinite(oh) && d_isfinite(ou) && d_isfinite(ov) && d_isfinite(zo));
        };
        // z_b (and G) entering the Exner update: the input's, or on ring cells the values of
        // the first boundary application
        auto ring_at = [&](int r) __attribute__((always_inline)) {  // slot of a ring cell, -1 elsewhere
            if (INTERIOR || idx < lo - 1 || idx > hi + 1 || !(r == 0 || r == ny - 1 || c == 0 || c == nx - 1)) return -1;
            return r == 0 ? idx : (r == ny - 1 ? pw + idx : 2 * pw + (c == 0 ? 0 : sr) + r - (R0 - 2));
        };
        auto bed = [&](int r) __attribute__((always_inline)) {
            const int s = ring_at(r);
            return s >= 0 ? slot_zb[s] : __ldg(a.zb + ((unsigned)r * upitch + (unsigned)c));
        };
        auto g_in = [&](int r) __attribute__((always_inline)) {
            const int s = ring_at(r);
            return s >= 0 ? slot_g[s] : __ldg(a.G + ((unsigned)r * upitch + (unsigned)c));
        };
        auto nod = [&](int r) __attribute__((always_inline)) {
            return HAS_MASK && colok && __ldg(a.nodata + ((unsigned)r * upitch + (unsigned)c)) != 0;
        };
        // Below the Shields threshold G is 0 and every Exner flux is 0 (q = G |u|^2 u): a warp
        // none of whose cells (its rows and the ones next to them) carries sediment leaves z_b
        // as it is.  Exact in both precisions: the skipped fluxes are +-0, and a NaN G is not 0.
        bool sediment = false;
        if (p0 < p1) {
            for (int r = max(p0 - 1, 0); r < min(p1 + 1, ny); ++r) {
                const int k = sidx(r, idx);
                if constexpr (MPM) sediment = sediment || (colok && mpm_may_move(Sh[k], Su[k], Sv[k], a.sed));
                else sediment = sediment || (colok && !(const_grass(Sh[k], g_in(r), nod(r)) == T(0)));
            }
            sediment = __any_sync(FULL, sediment);
        }
        if (!sediment) {
            if (out_col) {
                T zn[U];
#pragma unroll
                for (int u = 0; u < U; ++u) zn[u] = p0 + u < p1 ? bed(p0 + u) : T(0);
#pragma unroll 1
                for (int p = p0; p < p1; p += U) {  // the next U rows' loads are in flight while U rows are stored
                    Partner<T> q[U];
                    T zb[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        q[u] = qn[u];
                        zb[u] = zn[u];
                        qn[u] = partner(p + U + u);
                        zn[u] = p + U + u < p1 ? bed(p + U + u) : T(0);
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
                        if (p + u < p1) {
                            const int k = sidx(p + u, idx);
                            finish(p + u, Sh[k], Su[k], Sv[k], zb[u], T(0), q[u]);
                        }
                }
            }
        } else {
            T cu = T(0), cv = T(0), nu = T(0), nv = T(0);  // hu, hv of the current and the next row
            struct Bed { T zb, g; bool m; };  // what a row's cell needs from HBM, read a row ahead
            auto fetch = [&](int r) __attribute__((always_inline)) {
                Bed b{T(0), T(0), false};
                if ((INTERIOR || colok) && r < ny) {
                    b.zb = bed(r);
                    if (!MPM) b.g = g_in(r);
                    b.m = nod(r);
                }
                return b;
            };
            auto ecell = [&](int r, const Bed& b, T& hu, T& hv) __attribute__((always_inline)) {
                T h = T(0);
                hu = hv = T(0);
                if (INTERIOR || colok) {
                    const int k = sidx(r, idx);
                    h = Sh[k];
                    hu = Su[k];
                    hv = Sv[k];
                }
                const T G = MPM ? mpm_grass(h, hu, hv, b.m, a.sed) : const_grass(h, b.g, b.m);
                return make_ecell(h, hu, hv, b.zb, G);
            };
            int p = max(p0 - 1, 0);
            bool m = false, mnext = false;
            Bed b = fetch(p), bn = fetch(p + 1);
            Partner<T> q = qn[0];  // row p0
            ECell<T> e = ecell(p, b, cu, cv);
            m = b.m;
            T fn = T(0);
#pragma unroll 1
            for (; p < p1; ++p) {
                // in flight during this row's faces: the bed of row p+2, the partner of row p+1
                b = bn;
                mnext = b.m;
                if (p + 1 < p1) bn = fetch(p + 2);
                const Partner<T> qp = q;
                if (p >= p0) q = partner(p + 1);
                ECell<T> es{};
                const bool south = p + 1 < ny;
                if (south) es = ecell(p + 1, b, nu, nv);
                T fs = T(0);
                if (south) {
                    const bool act = colok && exner_active(e, es, m, mnext);
                    const T F = exner_face<T, true>(e, es);
                    fs = act ? F : T(0);
                    if constexpr (BUD && !INTERIOR) {
                        const int ps = p + 1;
                        if (act && out_col && (ps == 1 || ps == ny - 1) && ps >= p0 && ps < p1 && c >= 1 && c <= nx - 2)
                            budz += ps == 1 ? -(double)fs : (double)fs;
                    }
                }
                if (p >= p0) {
                    T xe = T(0);
                    const ECell<T> ee = shfl_down_ecell(e);
                    const bool me = HAS_MASK ? (__shfl_down_sync(FULL, (int)m, 1) != 0) : false;
                    const bool act = has_e && exner_active(e, ee, m, me);
                    const T Fx = exner_face<T, false>(e, ee);
                    const T F = act ? Fx : T(0);
                    if constexpr (BUD && !INTERIOR) {
                        if (act && out_col && p >= 1 && p <= ny - 2 && (c == 0 || c == nx - 2))
                            budz += c == 0 ? -(double)F : (double)F;
                    }
                    const T Fw = __shfl_up_sync(FULL, F, 1);
                    const bool wact = (__shfl_up_sync(FULL, (int)act, 1) != 0) && lane > 0;
                    // roe_exner.py:710-711: -F of the west face first, then +F of the east face
                    if (wact) xe = xe + (-Fw);
                    if (act) xe = xe + F;
                    T acc = xe;
                    acc = acc + (-fn);  // north face (roe_exner.py:712)
                    acc = acc + fs;     // south face (roe_exner.py:713)
                    T zo;
                    if constexpr (is_f32<T>()) zo = e.zb - dtdx * acc;
                    else zo = e.zb - dt * acc / dx;
                    finish(p, e.h, cu, cv, zo, e.G, qp);
                }
                fn = fs;
                e = es;
                cu = nu;
                cv = nv;
                m = mnext;
            }
        }
    }

    // ================= second boundary application and stores of the owned ring cells
    if (ring_tile) {
        __syncthreads();
        for (int k = threadIdx.x; k < nslots; k += blockDim.x) {
            int r, j;
            if (!slot_cell(k, r, j) || r < R0 || r >= R1 || j < lo || j > hi) continue;
            const pxb_ring_recipe rc = recipe(r, j);
            T oh, ou, ov;
            // a donor in the same row contributes its first-pass value; a donor in another
            // row is never a hydro boundary cell (checked at plan creation)
            apply_hydro(rc, sidx(r, j), oh, ou, ov);
            // position of the cell among the edge rows / columns, and its donors' positions
            int at, dz = 0, dg = 0;
            if (k < 2 * pw) {
                at = (r == 0 ? 0 : 3) * pw + j;
                dz = rc.zb_dy * pw + rc.zb_dx;
                dg = rc.g_dy * pw + rc.g_dx;
            } else {  // side columns: donors lie in the same row
                at = 4 * pw + (cstart + j == 0 ? 0 : 3) * sr + r - (R0 - 2);
                dz = rc.zb_dx * sr;
                dg = rc.g_dx * sr;
            }
            T zo = edge_z[(rc.flags & 8u) ? at + dz : at], go = edge_g[(rc.flags & 16u) ? at + dg : at];
            const unsigned i = (unsigned)r * upitch + (unsigned)(cstart + j);
            if (AVG) {
                oh = T(0.5) * a.ah[i] + T(0.5) * oh;
                ou = T(0.5) * a.ahu[i] + T(0.5) * ou;
                ov = T(0.5) * a.ahv[i] + T(0.5) * ov;
                zo = T(0.5) * a.azb[i] + T(0.5) * zo;
                if (a.oG) go = T(0.5) * a.aG[i] + T(0.5) * go;
            }
            a.oh[i] = oh;
            a.ohu[i] = ou;
            a.ohv[i] = ov;
            a.ozb[i] = zo;
            if (a.oG) a.oG[i] = go;
            bad |= !(d_isfinite(oh) && d_isfinite(ou) && d_isfinite(ov) && d_isfinite(zo));
        }
    }
    if constexpr (BUD) {  // this tile's outflow: warps in order, each summed in a fixed order
        __shared__ double part[2][32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            budh += __shfl_down_sync(FULL, budh, o);
            budz += __shfl_down_sync(FULL, budz, o);
        }
        if (lane == 0) {
            part[0][warp] = budh;
            part[1][warp] = budz;
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            double s = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += part[threadIdx.x][w];
            a.bud[2 * (size_t)tile + threadIdx.x] = s;
        }
    }
}

// Whether a tile lies away from the grid's boundary (see re_stage_tile).
template <class T>
__device__ __forceinline__ bool stage_tile_interior(const REStageArgs<T>& a, const int tile) {
    const int band = tile / a.nstrips, strip = tile - band * a.nstrips;
    return strip > 0 && strip < a.nstrips - 1 && band > 0 && band < a.nbands - 1;
}

template <class T>
__device__ __forceinline__ T* stage_shared() {
    extern __shared__ __align__(16) unsigned char stage_smem_raw[];
    return reinterpret_cast<T*>(stage_smem_raw);
}

template <class T, bool MPM, bool HAS_MASK, bool AVG, bool BUD = false>
__global__ void __launch_bounds__(stage_max_threads(sizeof(T)), stage_min_blocks(sizeof(T)))
    re_stage_kernel(const __grid_constant__ REStageArgs<T> a) {
    bool bad = false;
    const int tile = blockIdx.x;
    if (stage_tile_interior(a, tile)) re_stage_tile<T, MPM, HAS_MASK, AVG, BUD, true>(a, tile, stage_shared<T>(), bad);
    else re_stage_tile<T, MPM, HAS_MASK, AVG, BUD, false>(a, tile, stage_shared<T>(), bad);
    if (bad) atomicOr(a.err, 1);
}

}  // namespace pxb
