// Plain Roe shallow-water step (no Exner): PyExner src/PyExner/solvers/kernels/roe.py
// and src/PyExner/solvers/roe_solver.py.
//
// A block computes a tile of 16 x 8 cells: one thread per face of the tile into shared
// memory, then one thread per cell sums its four faces; ring cells with boundary recipes
// take their donor's update from shared memory, so the stage is one launch.  The
// configuration this solver is used for is small (258 x 258, float64): four threads per cell
// evaluated every face twice (and the donors' faces again), and a face's seven quotients and
// power took 64 registers with spills.  Bound by the float64 pipe and the length of a face's
// chain; us per SSPRK2 step with its dt, before -> after: float64 256^2 72 -> 29, 700^2 299 ->
// 112; float32 256^2 39 -> 21, 1000^2 299 -> 145.
#pragma once
#include "pxb_device.cuh"

namespace pxb {

template <class T>
struct RoeArgs {
    int ny, nx;
    long long pitch;
    T dx;
    const T *h, *hu, *hv, *z, *n;
    T *oh, *ohu, *ohv, *oz, *on;
    const T *ah, *ahu, *ahv, *az, *an;
    const T* dt;
    const pxb_ring_recipe* ring;
    int* err;
};

// Roe fluctuations with the wet/dry thrust and beta limiter (roe.py:32-249).  YF (the
// y-face orientation) is a runtime flag, so that the warp with both the last x-faces and the
// first y-faces of a tile runs one code path.
template <class T>
__device__ __forceinline__ void roe_plain_face(T hi, T hui, T hvi, T zi, T ni, T hj, T huj, T hvj, T zj, T nj, T dx,
                                               const bool YF, T P[3], T M[3]) {
    const T DRY = T(DRY_TOL);
    hi = hi > DRY ? hi : T(0);
    hj = hj > DRY ? hj : T(0);
    const T sqi = d_sqrt(hi), sqj = d_sqrt(hj);
    const DivBy<T> by_hi(hi), by_hj(hj);
    const T ui = hi > T(0) ? by_hi(hui) : T(0);
    const T vi = hi > T(0) ? by_hi(hvi) : T(0);
    const T uj = hj > T(0) ? by_hj(huj) : T(0);
    const T vj = hj > T(0) ? by_hj(hvj) : T(0);
    const T uhi = YF ? -vi : ui, vhi = YF ? ui : vi;
    const T uhj = YF ? -vj : uj, vhj = YF ? uj : vj;
    const T hsum = T(0.5) * (hi + hj);
    const T ht = hsum > DRY ? hsum : T(0);
    const T ct = d_sqrt(T(G_ACC) * ht);
    const DivBy<T> by_sq(sqi + sqj);
    const T ut = by_sq(uhi * sqi + uhj * sqj);
    const T vt = by_sq(vhi * sqi + vhj * sqj);
    T l1 = ut - ct;
    const T l2 = ut;
    T l3 = ut + ct;
    // Harten-Hyman: the fixed speed replaces lambda, then the entropy speed uses it (roe.py:77-92)
    T lE1 = T(0), lE3 = T(0);
    {
        const T ei = uhi - d_sqrt(T(G_ACC) * hi), ej = uhj - d_sqrt(T(G_ACC) * hj);
        const bool m = (ei < T(0)) && (ej > T(0));
        if (m) {
            l1 = ei * (ej - l1) / ((ej - ei) + T(VEL_TOL));
            lE1 = l1 - ei * (ej - l1) / ((ej - ei) + T(VEL_TOL));
        }
    }
    {
        const T ei = uhi + d_sqrt(T(G_ACC) * hi), ej = uhj + d_sqrt(T(G_ACC) * hj);
        const bool m = (ei < T(0)) && (ej > T(0));
        if (m) {
            l3 = ej * (l3 - ei) / ((ej - ei) + T(VEL_TOL));
            lE3 = l3 - ej * (l3 - ei) / ((ej - ei) + T(VEL_TOL));
        }
    }
    const T den = l1 - l3 + T(VEL_TOL);
    // (with ct = 0 the second wave is not a number, whichever way p10 comes out: b2 below)
    const DivBy<T> by_den(den), by_ct(ct);
    const T p00 = by_den(-l3), p01 = by_den(T(1));
    const T p10 = by_ct(-vt), p12 = T(1) / ct;
    const T p20 = by_den(l1), p21 = -p01;
    const T dh = hj - hi;
    const T dhu = hj * uhj - hi * uhi;
    const T dhv = hj * vhj - hi * vhi;
    // P^-1 dU accumulated over the inner index in order (roe.py:127)
    const T a1 = p00 * dh + p01 * dhu + T(0) * dhv;
    const T a2 = p10 * dh + T(0) * dhu + p12 * dhv;
    const T a3 = p20 * dh + p21 * dhu + T(0) * dhv;
    const T dz = zj - zi;
    const T di = hi + zi, dj = hj + zj;
    const T dd = dj - di;
    const T thrust_a = -T(G_ACC) * ht * dz;
    const bool k1 = (dz >= T(0)) && (di < zj);
    const bool k2 = (dz < T(0)) && (dj < zi);
    const T dzt = k1 ? hi : (k2 ? hj : dz);
    const T hr = dz >= T(0) ? hi : hj;
    const T thrust_b = -T(G_ACC) * (hr - T(0.5) * fabs(dzt)) * dzt;
    const bool mt = (dz * dd >= T(0)) && (ut * dz > T(0));
    const T thrust = mt ? nan_max(thrust_a, thrust_b) : thrust_b;
    const T nt = T(0.5) * (ni + nj);
    const T sf = (nt * nt * d_sqrt(ut * ut + vt * vt) * ut) / clamp_lo(d_pow43(ht), T(DRY_TOL));
    const T tau = T(G_ACC) * ht * sf * dx;
    const T T1 = thrust - tau;
    // P^-1 (0, T1, 0) (roe.py:159-165)
    T b1 = p00 * T(0) + p01 * T1 + T(0) * T(0);
    const T b2 = p10 * T(0) + T(0) * T1 + p12 * T(0);
    T b3 = p20 * T(0) + p21 * T1 + T(0) * T(0);
    const T hs1 = hi + a1 - (b1 / l1);
    const T hs3 = hj - a3 + (b3 / l3);
    const bool neg1 = (hs1 < T(0)) && (hs3 > T(0)), neg3 = (hs1 > T(0)) && (hs3 < T(0));
    if (neg1 || neg3) {
        const T b1min = -(hi + a1) * fabs(l1);
        const T b3min = -(hi - a1) * fabs(l3);
        const T dtf = dx / nan_max(nan_max(fabs(l1), fabs(l2)), fabs(l3));
        if (neg1) {
            const T dt1s = (dx / T(2) * l1) * (hi / (hi - hs1 + T(VEL_TOL)));
            if (dt1s < dtf) {
                b1 = (-b1min >= b3min) ? b1min : b1;
                b3 = -b1;
            }
        } else {
            const T dt3s = (dx / T(2) * l3) * (hj / (hj - hs3 + T(VEL_TOL)));
            if (dt3s < dtf) {
                b3 = (-b3min >= b3min) ? b1min : b3;
                b1 = -b3;
            }
        }
    }
    const bool mk1 = (hi < DRY) && (hs1 < T(0));
    const bool mk2 = (hj < DRY) && (hs3 < T(0));
    T p0 = 0, p1 = 0, p2 = 0, n0 = 0, n1 = 0, n2 = 0;
    const T lam[3] = {l1, l2, l3};
    const T alp[3] = {a1, a2, a3};
    const T bet[3] = {b1, b2, b3};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const T w = lam[k] * alp[k] - bet[k];
        const T f0 = (k == 1) ? w * T(0) : w;
        const T f1 = (k == 0) ? w * l1 : (k == 2 ? w * l3 : w * T(0));
        const T f2 = (k == 1) ? w * ct : w * vt;
        const bool pos = mk2 ? false : (mk1 ? true : (lam[k] > T(0)));
        const bool neg = mk2 ? true : (mk1 ? false : (lam[k] <= T(0)));
        if (pos) { p0 = p0 + f0; p1 = p1 + f1; p2 = p2 + f2; }
        if (neg) { n0 = n0 + f0; n1 = n1 + f1; n2 = n2 + f2; }
    }
    {
        const T e = lE1 * a1;
        if (lE1 > T(0)) { p0 = p0 + e; p1 = p1 + e * l1; p2 = p2 + e * vt; }
        else if (lE1 <= T(0)) { n0 = n0 + e; n1 = n1 + e * l1; n2 = n2 + e * vt; }
    }
    {
        const T e = lE3 * a3;
        if (lE3 > T(0)) { p0 = p0 + e; p1 = p1 + e * l3; p2 = p2 + e * vt; }
        else if (lE3 <= T(0)) { n0 = n0 + e; n1 = n1 + e * l3; n2 = n2 + e * vt; }
    }
    if (YF) {
        P[0] = p0; P[1] = p2; P[2] = -p1;
        M[0] = n0; M[1] = n2; M[2] = -n1;
    } else {
        P[0] = p0; P[1] = p1; P[2] = p2;
        M[0] = n0; M[1] = n1; M[2] = n2;
    }
}

// The larger of the two speeds of compute_dt for plain Roe (roe.py:13-30) at one cell,
// |u| + c + VEL_TOL and |v| + c + VEL_TOL, as an IEEE bit pattern (speeds are positive or
// NaN, so unsigned order is float order and NaN wins).
template <class T>
__device__ __forceinline__ unsigned long long roe_cell_speed_bits(T h0, T hu0, T hv0) {
    const bool wet = h0 > T(DRY_TOL);
    const T h = wet ? h0 : T(0);
    const T hv = wet ? hv0 : T(0);
    const T hu = wet ? hu0 : T(0);
    const T u = hu / (h + T(DRY_TOL));
    const T v = hv / (h + T(DRY_TOL));
    const T cc = d_sqrt(T(G_ACC) * h);
    const T sx = fabs(u) + cc + T(VEL_TOL);
    const T sy = fabs(v) + cc + T(VEL_TOL);
    const unsigned long long bx = speed_bits(sx), by = speed_bits(sy);
    return bx > by ? bx : by;
}

// Max over the launch of the threads' speed bits (warp max, block max through shared
// memory, one atomicMax per block), and the last block to finish turns it into
// dt = cfl * dx / smax (no floor), logs it and resets the accumulator.  Every thread of
// every block calls it once, at its end.
template <class T>
__device__ __forceinline__ void roe_dt_reduce(unsigned long long best, CflScratch* scr, T cfl, T dx, T* dt_out,
                                              T* dt_log) {
    const int lane = threadIdx.x & 31;
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(FULL, best, o);
        best = other > best ? other : best;
    }
    __shared__ unsigned long long wmax[32];
    if (lane == 0) wmax[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < (int)((blockDim.x + 31) >> 5); ++w) best = wmax[w] > best ? wmax[w] : best;
    if (best != 0ull) atomicMax(&scr->maxbits, best);
    __threadfence();  // the block's maximum before its ticket
    const unsigned int ticket = atomicAdd(&scr->done, 1u);
    if (ticket != gridDim.x - 1) return;
    __threadfence();
    const unsigned long long bits = atomicAdd(&scr->maxbits, 0ull);
    const T smax = bits_speed(bits, T(0));
    const T dt = cfl * (dx / smax);
    *dt_out = dt;
    if (dt_log) dt_log[scr->step] = dt;
    scr->step += 1;
    if (!d_isfinite(dt)) scr->err |= 2;
    scr->maxbits = 0ull;
    scr->done = 0u;
    __threadfence();
}

// Tile of a block: at most ROE_TX x ROE_TY cells; the tiles of a row or column of tiles
// differ by at most one cell and have at least two, so that a ring cell and its donors
// share one.
constexpr int ROE_TX = 16, ROE_TY = 8;
constexpr int ROE_XF = (ROE_TX + 1) * ROE_TY, ROE_YF = ROE_TX * (ROE_TY + 1);  // x-faces, y-faces
constexpr int ROE_THREADS = (ROE_XF + ROE_YF + 31) / 32 * 32;
static inline __host__ __device__ int roe_tiles(int n, int t) { return n > t ? (n + t - 1) / t : 1; }

// Resident blocks per SM the stage is register-limited to (tuning knob): 4 (56 registers) takes
// 29.1 us per step at 256^2 and 112 at 700^2 in float64, 3: 31.1 and 117, 2: 31.1 and 138.
#ifndef PXB_ROE_MIN_BLOCKS
#define PXB_ROE_MIN_BLOCKS 4
#endif

// One stage (roe_solver.py:40-54): update (roe.py:251-315), then the handlers.
template <class T, bool AVG>
__global__ void __launch_bounds__(ROE_THREADS, PXB_ROE_MIN_BLOCKS) roe_stage_kernel(const __grid_constant__ RoeArgs<T> a) {
    __shared__ T fx[6][ROE_XF], fy[6][ROE_YF], up[3][ROE_TX * ROE_TY];  // faces: upwP, upwM
    const int ntx = roe_tiles(a.nx, ROE_TX), nty = roe_tiles(a.ny, ROE_TY);
    const int by = blockIdx.x / ntx, bx = blockIdx.x - by * ntx;
    const int c0 = (int)((long long)a.nx * bx / ntx), c1 = (int)((long long)a.nx * (bx + 1) / ntx);
    const int r0 = (int)((long long)a.ny * by / nty), r1 = (int)((long long)a.ny * (by + 1) / nty);
    const T dt = *a.dt;
    const int t = threadIdx.x;
    // x-face f of a row lies west of column c0 + f, y-face f of a column north of row r0 + f
    const bool yf = t >= ROE_XF;
    const int k = yf ? t - ROE_XF : t;
    const int row = yf ? k / ROE_TX : k / (ROE_TX + 1), col = yf ? k - row * ROE_TX : k - row * (ROE_TX + 1);
    const int rj = r0 + row, cj = c0 + col, ri = yf ? rj - 1 : rj, ci = yf ? cj : cj - 1;
    const bool face = t < ROE_XF + ROE_YF && (yf ? (cj < c1 && rj <= r1 && ri >= 0 && rj < a.ny)
                                                 : (rj < r1 && cj <= c1 && ci >= 0 && cj < a.nx));
    if (face) {
        const long long i = (long long)ri * a.pitch + ci, j = (long long)rj * a.pitch + cj;
        T P[3], M[3];
        roe_plain_face<T>(a.h[i], a.hu[i], a.hv[i], a.z[i], a.n[i], a.h[j], a.hu[j], a.hv[j], a.z[j], a.n[j], a.dx, yf, P, M);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            (yf ? fy[m][k] : fx[m][k]) = P[m];
            (yf ? fy[3 + m][k] : fx[3 + m][k]) = M[m];
        }
    }
    __syncthreads();
    const int tr = t / ROE_TX, tc = t - tr * ROE_TX, r = r0 + tr, c = c0 + tc;
    const bool cell = t < ROE_TX * ROE_TY && r < r1 && c < c1;
    const long long i = (long long)r * a.pitch + c;
    T u[3] = {T(0), T(0), T(0)};
    if (cell) {
        // scatter order of roe.py:296-299: east upwM, west upwP, south upwM, north upwP
        T f[3] = {T(0), T(0), T(0)};
        const int xw = tr * (ROE_TX + 1) + tc, yn = tr * ROE_TX + tc;
#pragma unroll
        for (int m = 0; m < 3; ++m) {
            if (c + 1 < a.nx) f[m] = f[m] + fx[3 + m][xw + 1];
            if (c >= 1) f[m] = f[m] + fx[m][xw];
            if (r + 1 < a.ny) f[m] = f[m] + fy[3 + m][yn + ROE_TX];
            if (r >= 1) f[m] = f[m] + fy[m][yn];
        }
        const DivBy<T> by_dx(a.dx);
        u[0] = a.h[i] - by_dx(dt * f[0]);
        u[1] = a.hu[i] - by_dx(dt * f[1]);
        u[2] = a.hv[i] - by_dx(dt * f[2]);
#pragma unroll
        for (int m = 0; m < 3; ++m) up[m][t] = u[m];
    }
    __syncthreads();
    if (!cell) return;
    // Roe handlers write h, z and n from one donor (flags bit 0) and the momentum from
    // another (bit 1: a 2x2 map of the donor's, or constants with bit 2).
    const bool on_ring = (r == 0) || (r == a.ny - 1) || (c == 0) || (c == a.nx - 1);
    if (on_ring) {
        T zo = a.z[i], no = a.n[i];
        if (a.ring != nullptr) {
            const pxb_ring_recipe& rc = a.ring[ring_slot(r, c, a.ny, a.nx)];
            if (rc.flags & 1u) {
                u[0] = up[0][t + rc.h_dy * ROE_TX + rc.h_dx];
                const long long j = (long long)(r + rc.h_dy) * a.pitch + (c + rc.h_dx);
                zo = a.z[j];
                no = a.n[j];
            }
            if (rc.flags & 4u) {
                u[1] = T(rc.m[0]);
                u[2] = T(rc.m[1]);
            } else if (rc.flags & 2u) {
                const int d = t + rc.m_dy * ROE_TX + rc.m_dx;
                const T du = up[1][d], dv = up[2][d];
                u[1] = T(rc.m[0]) * du + T(rc.m[1]) * dv;
                u[2] = T(rc.m[2]) * du + T(rc.m[3]) * dv;
            }
        }
        if (AVG) {
            zo = T(0.5) * a.az[i] + T(0.5) * zo;
            no = T(0.5) * a.an[i] + T(0.5) * no;
        }
        a.oz[i] = zo;
        a.on[i] = no;
    }
    if (AVG) {
        u[0] = T(0.5) * a.ah[i] + T(0.5) * u[0];
        u[1] = T(0.5) * a.ahu[i] + T(0.5) * u[1];
        u[2] = T(0.5) * a.ahv[i] + T(0.5) * u[2];
    }
    a.oh[i] = u[0];
    a.ohu[i] = u[1];
    a.ohv[i] = u[2];
    if (!(d_isfinite(u[0]) && d_isfinite(u[1]) && d_isfinite(u[2]))) atomicOr(a.err, 1);
}

// compute_dt for plain Roe (roe.py:13-30): cfl * dx / max over ALL cells of
// (|u| + c + VEL_TOL) and (|v| + c + VEL_TOL); no floor.
template <class T>
__global__ void __launch_bounds__(256) roe_cfl_kernel(const CflArgs<T> a) {
    unsigned long long best = 0ull;
    const long long ncell = (long long)a.ny * a.nx;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < ncell; k += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(k / a.nx), c = (int)(k - (long long)r * a.nx);
        const long long i = (long long)r * a.pitch + c;
        const unsigned long long b = roe_cell_speed_bits(a.h[i], a.hu[i], a.hv[i]);
        best = b > best ? b : best;
    }
    roe_dt_reduce<T>(best, a.scr, a.cfl, a.dx, a.dt_out, a.dt_log);
}

}  // namespace pxb
