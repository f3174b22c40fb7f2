// Reverse-mode (adjoint) kernels of the float64 Roe-Exner stage and of the CFL step.
//
// A stage is, in the reference's order (roe_exner_solver.py:80-116):
//   U1 = U - dt/dx * sum of face fluctuations(U)          hydro (roe_exner.py:535-612)
//   momentum corrections (zeroing masks)                    (:14-62)
//   handlers                                                (boundary_registry.py:183-187)
//   G = grass(h, hu, hv) or the constant pass-through      (:85-140)
//   zb2 = zb1 - dt/dx * sum of Exner face fluxes            (:665-717)
//   handlers
// and the SSPRK2 average for the second stage.  The adjoint runs these backwards.  The hydro
// faces and the MPM grass factor are differentiated by hand (adj_exner_hydro_face restates
// roe_exner_face, mpm_gradient restates mpm_grass: a change to one belongs in the other; the
// transpose tests compare them through the tangent model, which runs the forward formulas).
// The Exner and CFL faces are evaluated by the forward formulas on DualN numbers seeded with
// the cells' inputs.  Masks and branches (wet/dry, activity, upwinding, the correction
// zeroing) are taken from the forward values and carry no derivative.
// Handlers are linear in the state for every kind except ConstantOutflux (refused):
// their adjoint moves the boundary cells' adjoints to the donors (scatter-add).
#pragma once
// pxb_device.cuh first: its templates must see the standard fabs at their definition;
// the dual types bring their own overloads through argument-dependent lookup.
#include "pxb_device.cuh"
#include "init_bc.cuh"
#include "adjoint_args.cuh"
#include "dualn.cuh"
#include "re_cfl.cuh"  // cfl_bound

namespace pxb {


__device__ __forceinline__ bool adj_cell(int ny, int nx, long long pitch, int& r, int& c, long long& i) {
    c = blockIdx.x * blockDim.x + threadIdx.x;
    r = blockIdx.y * blockDim.y + threadIdx.y;
    if (r >= ny || c >= nx) return false;
    i = (long long)r * pitch + c;
    return true;
}

__device__ __forceinline__ bool adj_nodata(const uint8_t* m, long long i) { return m ? m[i] != 0 : false; }

// Sum over the block of each of N values, one atomic per value and block: atomics of all
// warps of a 512^2 grid on one address took about 60 us.  Every thread of a block of up to
// 1024 calls it once.
template <int N>
__device__ __forceinline__ void adj_sum_add(double* dst, const double (&v)[N]) {
    __shared__ double part[N][32];
    const int tid = threadIdx.x + blockDim.x * threadIdx.y, warp = tid >> 5, nw = (blockDim.x * blockDim.y) >> 5;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        double x = v[q];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
        if ((tid & 31) == 0) part[q][warp] = x;
    }
    __syncthreads();
    if (tid < N) {
        double x = 0.0;
        for (int w = 0; w < nw; ++w) x += part[tid][w];
        if (x != 0.0) atomicAdd(dst + tid, x);
    }
}
__device__ __forceinline__ void adj_dt_add(double* dst, double v) {
    const double x[1] = {v};
    adj_sum_add<1>(dst, x);
}

// SSPRK2 average / plain store: S = scale * out_adj; with `avg`, avg_adj = 0.5 * out_adj.
__global__ void adj_store_kernel(int ny, int nx, long long pitch, double scale, const double* oh, const double* ohu,
                                 const double* ohv, const double* ozb, const double* oG, double* Sh, double* Shu,
                                 double* Shv, double* Szb, double* SG, double* Ah, double* Ahu, double* Ahv, double* Azb,
                                 double* AG) {
    int r, c;
    long long i;
    if (!adj_cell(ny, nx, pitch, r, c, i)) return;
    const double a[5] = {oh[i], ohu[i], ohv[i], ozb[i], oG[i]};
    Sh[i] = scale * a[0];
    Shu[i] = scale * a[1];
    Shv[i] = scale * a[2];
    Szb[i] = scale * a[3];
    SG[i] = scale * a[4];
    if (Ah) {
        Ah[i] = 0.5 * a[0];
        Ahu[i] = 0.5 * a[1];
        Ahv[i] = 0.5 * a[2];
        Azb[i] = 0.5 * a[3];
        AG[i] = 0.5 * a[4];
    }
}

// Exner update backwards: T = S (identity paths) + face terms; dt adjoint.
__global__ void __launch_bounds__(256) adj_exner_kernel(const AdjArgs a) {
    int r, c;
    long long i;
    const bool in = adj_cell(a.ny, a.nx, a.pitch, r, c, i);
    double add_dt = 0.0;
    if (in) {
        using D = DualN<5>;
        const double dt = *a.dt, dx = a.dx;
        auto ecell = [&](long long k) { return make_ecell(a.sh[k], a.shu[k], a.shv[k], a.szb[k], a.sG[k]); };
        const ECell<double> C = ecell(i);
        const ECell<D> Cd = make_ecell(D::seed(a.sh[i], 0), D::seed(a.shu[i], 1), D::seed(a.shv[i], 2),
                                       D::seed(a.szb[i], 3), D::seed(a.sG[i], 4));
        auto econst = [&](long long k) {
            return make_ecell(D(a.sh[k]), D(a.shu[k]), D(a.shv[k]), D(a.szb[k]), D(a.sG[k]));
        };
        const bool mC = adj_nodata(a.nodata, i);
        double g[5] = {0, 0, 0, 0, 0};
        double acc = 0.0;  // sum of the signed face fluxes of this cell (forward values)
        // face (I|J) with flux F: zb2[I] -= dt/dx F, zb2[J] += dt/dx F
        auto face = [&](long long k, bool cell_is_I, bool yf) {
            const ECell<double> N = ecell(k);
            const bool mk = adj_nodata(a.nodata, k);
            const bool act = cell_is_I ? exner_active(C, N, mC, mk) : exner_active(N, C, mk, mC);
            if (!act) return;
            const ECell<D> Nd = econst(k);
            D F;
            if (yf) F = cell_is_I ? exner_face<D, true>(Cd, Nd) : exner_face<D, true>(Nd, Cd);
            else F = cell_is_I ? exner_face<D, false>(Cd, Nd) : exner_face<D, false>(Nd, Cd);
            const double zI = cell_is_I ? a.Szb[i] : a.Szb[k], zJ = cell_is_I ? a.Szb[k] : a.Szb[i];
            const double Fbar = -dt / dx * (zI - zJ);
            for (int q = 0; q < 5; ++q) g[q] += Fbar * F.d[q];
            acc += cell_is_I ? F.v : -F.v;
        };
        if (c >= 1) face(i - 1, false, false);
        if (c + 1 < a.nx) face(i + 1, true, false);
        if (r >= 1) face(i - a.pitch, false, true);
        if (r + 1 < a.ny) face(i + a.pitch, true, true);
        (void)C;
        a.Th[i] = a.Sh[i] + g[0];
        a.Thu[i] = a.Shu[i] + g[1];
        a.Thv[i] = a.Shv[i] + g[2];
        a.Tzb[i] = a.Szb[i] + g[3];
        a.TG[i] = a.SG[i] + g[4];
        add_dt = a.Szb[i] * (-acc / dx);
    }
    adj_dt_add(a.dtbar, add_dt);
}

// Derivatives of the Meyer-Peter & Mueller grass factor of one cell (roe_exner.py:85-130):
// G = sum_k frac g1 g2 d / (1 - porosity) with d = theta - theta_c, g1 = n_p^3 sqrt(g) /
// ((s-1) sqrt(h)), g2 = 8 sqrt(d) / (theta^1.5 + 1e-5), theta = n_p^2 |u|^2 / ((s-1) d50
// h^(1/3)).  dh, dhu, dhv: with respect to the cell's planes; par[7] (PAR): with respect to
// the constants of the one class (n_p^2, (s-1) d50, theta_c, n_p^3 sqrt(g), s-1, fraction,
// 1 - porosity).  Zero at and below the threshold and in dry cells, as the clamps give.
template <bool PAR>
__device__ __forceinline__ void mpm_gradient(double h, double hu, double hv, const SedTable<double>& S, double& dh,
                                             double& dhu, double& dhv, double (&par)[7]) {
    dh = dhu = dhv = 0.0;
#pragma unroll
    for (int q = 0; q < 7; ++q) par[q] = 0.0;
    if (!(h > DRY_TOL)) return;
    const DivBy<double> by_h(h);
    const double u = by_h(hu), v = by_h(hv), vel2 = u * u + v * v, cb = cbrt(h), sqh = sqrt(h);
    for (int k = 0; k < S.n; ++k) {
        const SedT<double>& c = S.s[k];
        const double per = c.np2 / (c.sm1d * cb);  // theta per |u|^2
        const double theta = per * vel2, d = theta - c.thc;
        if (!(d > 0.0)) {  // (a NaN stays in the value, not in the derivatives of other cells)
            if (d != d) dh = dhu = dhv = d;
            continue;
        }
        const double rt = sqrt(theta), rd = sqrt(d), den = 1.0 / (theta * rt + 1e-5);
        const double g1 = c.np3sg / (c.sm1 * sqh), unit = g1 * 8.0 / S.one_minus_por, amp = c.frac * unit;
        const double G = amp * rd * d * den;
        const double g_d = 1.5 * amp * rd * den;                 // through d
        const double g_t = g_d - 1.5 * G * rt * den;             // through theta
        const double t_h = by_h(theta) * (-7.0 / 3.0), t_u = per * 2.0 * by_h(1.0) * g_t;
        dh += g_t * t_h - 0.5 * by_h(G);
        dhu += t_u * u;
        dhv += t_u * v;
        if (PAR) {
            par[0] = g_t * theta / c.np2;
            par[1] = -g_t * theta / c.sm1d;
            par[2] = -g_d;
            par[3] = G / c.np3sg;
            par[4] = -G / c.sm1;
            par[5] = unit * rd * d * den;  // (not by the fraction, which may be 0)
            par[6] = -G / S.one_minus_por;
        }
    }
}

// grass factor backwards, in place on T (G of the state after handlers 1 -> h, hu, hv);
// PAR: also the adjoint of the MPM constants of the single sediment class (a.tbar).  The
// derivatives are written out instead of taken from dual numbers with ten tangents.
template <bool PAR>
__global__ void __launch_bounds__(256) adj_grass_kernel(const AdjArgs a) {
    int r, c;
    long long i;
    const bool in = adj_cell(a.ny, a.nx, a.pitch, r, c, i);
    double tb[7] = {0, 0, 0, 0, 0, 0, 0};
    if (in) {
        const bool m = adj_nodata(a.nodata, i);
        const double gbar = a.TG[i];
        if (a.mpm) {
            if (!m) {
                double dh, dhu, dhv, par[7];
                mpm_gradient<PAR>(a.sh[i], a.shu[i], a.shv[i], a.sed, dh, dhu, dhv, par);
                a.Th[i] += gbar * dh;
                a.Thu[i] += gbar * dhu;
                a.Thv[i] += gbar * dhv;
                if (PAR)
#pragma unroll
                    for (int q = 0; q < 7; ++q) tb[q] = gbar * par[q];
            }
            a.TG[i] = 0.0;  // MPM recomputes G: the incoming G has no influence
        } else {
            a.TG[i] = (!m && a.sh[i] > DRY_TOL) ? gbar : 0.0;
        }
    }
    if constexpr (PAR) adj_sum_add<7>(a.tbar, tb);
}

// momentum corrections backwards, in place on T (interior cells)
__global__ void adj_corr_kernel(const AdjArgs a) {
    int r, c;
    long long i;
    if (!adj_cell(a.ny, a.nx, a.pitch, r, c, i)) return;
    if (r < 1 || r > a.ny - 2 || c < 1 || c > a.nx - 2) return;
    const double DRY = DRY_TOL;
    const long long E = i + 1, W = i - 1, N = i - a.pitch, S = i + a.pitch;
    const double eta = a.h1[i] + (a.z[i] + a.zb[i]);
    const bool stop_u = ((eta < a.z[E] + a.zb[E]) && (a.h1[E] < DRY)) || ((eta < a.z[W] + a.zb[W]) && (a.h1[W] < DRY)) ||
                        adj_nodata(a.nodata, E) || adj_nodata(a.nodata, W);
    const bool stop_v = ((eta < a.z[N] + a.zb[N]) && (a.h1[N] < DRY)) || ((eta < a.z[S] + a.zb[S]) && (a.h1[S] < DRY)) ||
                        adj_nodata(a.nodata, N) || adj_nodata(a.nodata, S);
    const bool active = (a.h1[i] > DRY) && !adj_nodata(a.nodata, i);
    if (!(active && !stop_u)) a.Thu[i] = 0.0;
    if (!(active && !stop_v)) a.Thv[i] = 0.0;
}

// Adjoints of the values of one cell that a Roe-Exner face reads (HCell).
struct HBar {
    double h, u, v, z, nb;  // clamped depth (with its square root and celerity), velocities, bed, n_b
};

// One face backwards (roe_exner_face): Pb, Mb are the adjoints of upwP and upwM; bI, bJ
// receive those of the two cells' values, P and M the fluctuations.  Branches (entropy fix,
// signs of the speeds, the floor of h^(4/3)) are the forward ones.
template <bool YF>
__device__ __forceinline__ void adj_exner_hydro_face(const HCell<double>& I, const HCell<double>& J, const double dx,
                                                     const double (&Pb)[3], const double (&Mb)[3], HBar& bI, HBar& bJ,
                                                     double (&P)[3], double (&M)[3]) {
    const double uI = YF ? -I.v : I.u, vI = YF ? I.u : I.v, uJ = YF ? -J.v : J.u, vJ = YF ? J.u : J.v;
    const double ht = 0.5 * (I.h + J.h), ct = sqrt(G_ACC * ht);
    const DivBy<double> by_den(I.sq + J.sq), by_c(ct);
    const double ut = by_den(uI * I.sq + uJ * J.sq), vt = by_den(vI * I.sq + vJ * J.sq);
    const double l1r = ut - ct, l3r = ut + ct;
    const double ei = uI - I.c, ej = uJ - J.c, fi = uI + I.c, fj = uJ + J.c;
    const bool m1 = ei < 0.0 && ej > 0.0, m3 = fi < 0.0 && fj > 0.0;
    double l1 = l1r, l3 = l3r, lE1 = 0.0, lE3 = 0.0;
    if (m1) {
        l1 = ei * (ej - l1r) / (ej - ei);
        lE1 = l1r - l1;
    }
    if (m3) {
        const double num = fj * (l3r - fi);
        lE3 = l3r - num / (fj - fi);
        l3 = num / ((fj - fi) + VEL_TOL);
    }
    const double dh = J.h - I.h, dhu = J.h * uJ - I.h * uI, dhv = J.h * vJ - I.h * vI, dz = J.zt - I.zt;
    const double a1 = -0.5 * by_c(-l3r * dh + dhu), a2 = by_c(-vt * dh + dhv), a3 = -0.5 * by_c(l1r * dh - dhu);
    const double nt = 0.5 * (I.nb + J.nb), speed = sqrt(ut * ut + vt * vt), cb = cbrt(ht);
    const double D43 = ht * cb;
    const bool floored = D43 < DRY_TOL;
    const double rD = 1.0 / (floored ? DRY_TOL : D43);
    const double sf = nt * nt * speed * ut * rD;
    const double thrust = -G_ACC * ht * dz, tau = G_ACC * ht * sf * dx;
    const double b1 = -0.5 * by_c(thrust - tau);
    const double w1 = l1 * a1 - b1, w2 = ut * a2, w3 = l3 * a3 + b1;
    // fluctuations and their adjoints in the face's frame (1: normal, 2: tangential)
    const double pb0 = Pb[0], pb1 = YF ? -Pb[2] : Pb[1], pb2 = YF ? Pb[1] : Pb[2];
    const double nb0 = Mb[0], nb1 = YF ? -Mb[2] : Mb[1], nb2 = YF ? Mb[1] : Mb[2];
    double p0 = 0, p1 = 0, p2 = 0, n0 = 0, n1 = 0, n2 = 0;
    double l1b = 0, l3b = 0, a1b = 0, a3b = 0, vtb = 0, b1b = 0, lE1b = 0, lE3b = 0;
    auto wave = [&](bool pos, double w, double l, double& lb) __attribute__((always_inline)) {  // -> adjoint of w
        (pos ? p0 : n0) += w;
        (pos ? p1 : n1) += w * l;
        (pos ? p2 : n2) += w * vt;
        const double B0 = pos ? pb0 : nb0, B1 = pos ? pb1 : nb1, B2 = pos ? pb2 : nb2;
        lb += B1 * w;
        vtb += B2 * w;
        return B0 + B1 * l + B2 * vt;
    };
    const double w1b = wave(l1 > 0.0, w1, l1, l1b);
    const double w3b = wave(l3 > 0.0, w3, l3, l3b);
    l1b += w1b * a1;
    a1b += w1b * l1;
    l3b += w3b * a3;
    a3b += w3b * l3;
    b1b += w3b - w1b;
    const bool s2 = ut > 0.0;
    (s2 ? p2 : n2) += w2 * ct;
    const double B2 = s2 ? pb2 : nb2, w2b = B2 * ct;
    double ctb = B2 * w2, utb = w2b * a2, l1rb = 0.0, l3rb = 0.0;
    const double a2b = w2b * ut;
    double uIb = 0, uJb = 0, cIb = 0, cJb = 0;
    if (m1) {
        const double eb = wave(lE1 > 0.0, lE1 * a1, l1, l1b);
        lE1b = eb * a1;
        a1b += eb * lE1;
        const double dd = 1.0 / (ej - ei), tb = l1b - lE1b;
        const double eib = tb * ((ej - l1r) + l1) * dd, ejb = tb * (ei - l1) * dd;
        l1rb += lE1b - tb * ei * dd;
        uIb += eib, cIb -= eib, uJb += ejb, cJb -= ejb;
    } else {
        l1rb += l1b;
    }
    if (m3) {
        const double eb = wave(lE3 > 0.0, lE3 * a3, l3, l3b);
        lE3b = eb * a3;
        a3b += eb * lE3;
        const double d0 = 1.0 / (fj - fi), d1 = 1.0 / ((fj - fi) + VEL_TOL), q = l3r - lE3;
        const double numb = l3b * d1 - lE3b * d0, d0b = lE3b * q * d0 - l3b * l3 * d1;
        const double fjb = numb * (l3r - fi) + d0b, fib = -numb * fj - d0b;
        l3rb += lE3b + numb * fj;
        uIb += fib, cIb += fib, uJb += fjb, cJb += fjb;
    } else {
        l3rb += l3b;
    }
    // wave strengths and the source
    const double y1 = -0.5 * by_c(a1b), y2 = by_c(a2b), y3 = -0.5 * by_c(a3b), yb = -0.5 * by_c(b1b);
    ctb -= by_c(a1b * a1 + a2b * a2 + a3b * a3 + b1b * b1);
    l3rb -= y1 * dh;
    l1rb += y3 * dh;
    vtb -= y2 * dh;
    const double dhb = -y1 * l3r - y2 * vt + y3 * l1r, dhub = y1 - y3, dhvb = y2;
    double htb = -yb * G_ACC * dz - yb * G_ACC * sf * dx;
    const double dzb = -yb * G_ACC * ht, sfb = -yb * G_ACC * ht * dx;
    const double ntb = sfb * 2.0 * nt * speed * ut * rD, spb = sfb * nt * nt * ut * rD;
    utb += sfb * nt * nt * speed * rD;
    if (!floored) htb -= sfb * sf * rD * (4.0 / 3.0) * cb;
    if (speed > 0.0) {
        const double k = spb / speed;
        utb += k * ut;
        vtb += k * vt;
    }
    utb += l1rb + l3rb;
    ctb += l3rb - l1rb;
    htb += 0.5 * G_ACC * by_c(ctb);
    const double yu = by_den(utb), yv = by_den(vtb);
    uIb += yu * I.sq - dhub * I.h;
    uJb += yu * J.sq + dhub * J.h;
    const double vIb = yv * I.sq - dhvb * I.h, vJb = yv * J.sq + dhvb * J.h;
    const double sIb = yu * (uI - ut) + yv * (vI - vt), sJb = yu * (uJ - ut) + yv * (vJ - vt);
    // sqrt(h) and sqrt(g h) of the cells back to their depths
    bI.h = 0.5 * htb - dhb - dhub * uI - dhvb * vI + 0.5 * sIb / I.sq + 0.5 * G_ACC * cIb / I.c;
    bJ.h = 0.5 * htb + dhb + dhub * uJ + dhvb * vJ + 0.5 * sJb / J.sq + 0.5 * G_ACC * cJb / J.c;
    bI.u = YF ? vIb : uIb;
    bI.v = YF ? -uIb : vIb;
    bJ.u = YF ? vJb : uJb;
    bJ.v = YF ? -uJb : vJb;
    bI.z = -dzb;
    bJ.z = dzb;
    bI.nb = bJ.nb = 0.5 * ntb;
    P[0] = p0, P[1] = YF ? p2 : p1, P[2] = YF ? -p1 : p2;
    M[0] = n0, M[1] = YF ? n2 : n1, M[2] = YF ? -n1 : n2;
}

// Tile of adj_hydro_kernel: at most 16 x 8 cells, one thread per face.
constexpr int ADJ_TX = 16, ADJ_TY = 8;
constexpr int ADJ_XF = (ADJ_TX + 1) * ADJ_TY, ADJ_YF = ADJ_TX * (ADJ_TY + 1);
constexpr int ADJ_THREADS = (ADJ_XF + ADJ_YF + 31) / 32 * 32;

// hydro update backwards: I += T (identity paths) + face terms; dt adjoint.  NB: also the
// adjoint of the cells' n_b (Manning friction of their faces), added to a.nbbar.  Every face
// of a tile is differentiated once, in reverse, for both of its cells; before, each cell
// evaluated its four faces on dual numbers with five tangents: 528 us at 512^2, 87 now.
// Bound by the float64 pipe.
#ifndef PXB_ADJ_MIN_BLOCKS
#define PXB_ADJ_MIN_BLOCKS 2
#endif
template <bool NB>
__global__ void __launch_bounds__(ADJ_THREADS, PXB_ADJ_MIN_BLOCKS) adj_hydro_kernel(const __grid_constant__ AdjArgs a) {
    __shared__ double fx[10][ADJ_XF], fy[10][ADJ_YF];  // adjoints of the first, then of the second cell
    const int t = threadIdx.x, c0 = blockIdx.x * ADJ_TX, r0 = blockIdx.y * ADJ_TY;
    const int c1 = min(a.nx, c0 + ADJ_TX), r1 = min(a.ny, r0 + ADJ_TY);
    const double dt = *a.dt, dx = a.dx, DRY = DRY_TOL;
    // x-face f of a row lies west of column c0 + f, y-face f of a column north of row r0 + f
    const bool yf = t >= ADJ_XF;
    const int k = yf ? t - ADJ_XF : t;
    const int row = yf ? k / ADJ_TX : k / (ADJ_TX + 1), col = yf ? k - row * ADJ_TX : k - row * (ADJ_TX + 1);
    const int rj = r0 + row, cj = c0 + col, ri = yf ? rj - 1 : rj, ci = yf ? cj : cj - 1;
    bool face = t < ADJ_XF + ADJ_YF && (yf ? (cj < c1 && rj <= r1 && ri >= 0 && rj < a.ny)
                                           : (rj < r1 && cj <= c1 && ci >= 0 && cj < a.nx));
    const long long i = (long long)ri * a.pitch + ci, j = (long long)rj * a.pitch + cj;
    if (face) face = ((a.h[i] > DRY) || (a.h[j] > DRY)) && !(adj_nodata(a.nodata, i) || adj_nodata(a.nodata, j));
    double add_dt = 0.0;
    HBar bI{0, 0, 0, 0, 0}, bJ{0, 0, 0, 0, 0};
    if (face) {
        const double k_ = -dt / dx;
        const double aI[3] = {a.Th[i], a.Thu[i], a.Thv[i]}, aJ[3] = {a.Th[j], a.Thu[j], a.Thv[j]};
        const double Pb[3] = {k_ * aJ[0], k_ * aJ[1], k_ * aJ[2]}, Mb[3] = {k_ * aI[0], k_ * aI[1], k_ * aI[2]};
        const HCell<double> I = make_hcell(a.h[i], a.hu[i], a.hv[i], a.zb[i], a.z[i], a.nb[i]);
        const HCell<double> J = make_hcell(a.h[j], a.hu[j], a.hv[j], a.zb[j], a.z[j], a.nb[j]);
        double P[3], M[3];
        if (yf) adj_exner_hydro_face<true>(I, J, dx, Pb, Mb, bI, bJ, P, M);
        else adj_exner_hydro_face<false>(I, J, dx, Pb, Mb, bI, bJ, P, M);
        // the tile of the second cell counts the face
        if (yf ? rj < r1 : cj < c1)
            add_dt = -((aI[0] * M[0] + aI[1] * M[1] + aI[2] * M[2]) + (aJ[0] * P[0] + aJ[1] * P[1] + aJ[2] * P[2])) / dx;
    }
    if (t < ADJ_XF + ADJ_YF) {
        const double v[10] = {bI.h, bI.u, bI.v, bI.z, bI.nb, bJ.h, bJ.u, bJ.v, bJ.z, bJ.nb};
#pragma unroll
        for (int m = 0; m < 10; ++m) (yf ? fy[m][k] : fx[m][k]) = v[m];
    }
    adj_dt_add(a.dtbar, add_dt);
    __syncthreads();
    const int tr = t / ADJ_TX, tc = t - tr * ADJ_TX, r = r0 + tr, c = c0 + tc;
    if (t >= ADJ_TX * ADJ_TY || r >= r1 || c >= c1) return;
    const int xw = tr * (ADJ_TX + 1) + tc, yn = tr * ADJ_TX + tc;
    double g[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {  // faces beyond the grid hold zeros
        g[m] = fx[m][xw + 1] + fx[5 + m][xw];
        g[m] = g[m] + fy[m][yn + ADJ_TX];
        g[m] = g[m] + fy[5 + m][yn];
    }
    // the clamps, velocities and the bed of make_hcell backwards
    const long long o = (long long)r * a.pitch + c;
    const double h = a.h[o], hc = clamp_lo(h, DRY);
    double gh = g[0], ghu = 0.0, ghv = 0.0;
    if (hc > DRY) {
        const DivBy<double> by_h(hc);
        ghu = by_h(g[1]);
        ghv = by_h(g[2]);
        gh -= ghu * by_h(a.hu[o]) + ghv * by_h(a.hv[o]);
    }
    if (h < DRY) gh = 0.0;
    a.Ih[o] += a.Th[o] + gh;
    a.Ihu[o] += a.Thu[o] + ghu;
    a.Ihv[o] += a.Thv[o] + ghv;
    a.Izb[o] += a.Tzb[o] + (a.zb[o] > SED_TOL ? g[3] : 0.0);
    a.IG[o] += a.TG[o];
    if constexpr (NB) a.nbbar[o] += g[4];
}

// ---------------------------------------------------------------- handlers backwards

// The adjoint of a boundary cell's fields that the handler writes, taken and cleared (they
// were overwritten); read past the L1, behind the atomics of the handler before.
__device__ __forceinline__ void adj_bc_take(const AdjBcSet& a, const AdjBcHandler& h, const long long b, double (&t)[6]) {
    const unsigned fm = bc_field_mask(h.kind);
    auto writes = [&](int s) { return ((fm >> s) & 1u) && a.f[s]; };
#pragma unroll
    for (int s = 0; s < 6; ++s) t[s] = writes(s) ? __ldcg(a.f[s] + b) : 0.0;
    // (all loads in flight before the first store, which might alias the next plane)
#pragma unroll
    for (int s = 0; s < 6; ++s)
        if (writes(s)) a.f[s][b] = 0.0;
}

// The donor receives the transposed Jacobian of the handler times the adjoints taken.
__device__ __forceinline__ void adj_bc_give(const AdjBcSet& a, const AdjBcHandler& h, const long long d, const double (&t)[6]) {
    auto add = [&](int s, double v) {
        if (a.f[s] && v != 0.0) atomicAdd(a.f[s] + d, v);
    };
    switch (h.kind) {
        case PXB_BC_RE_REFLECTIVE: {  // hu' = (-nx^2 + ny^2) hu - 2 nx ny hv, hv' = -2 nx ny hu + (nx^2 - ny^2) hv
            const double nx = h.nx, ny = h.ny;
            // forward: mom_n = hu nx + hv ny, mom_t = -hu ny + hv nx, hu' = -mom_n nx - mom_t ny,
            // hv' = -mom_n ny + mom_t nx
            const double bu = t[1], bv = t[2];
            const double bmn = -bu * nx - bv * ny, bmt = -bu * ny + bv * nx;
            add(0, t[0]);
            add(1, bmn * nx - bmt * ny);
            add(2, bmn * ny + bmt * nx);
            add(3, t[3]);
            add(5, t[5]);
            break;
        }
        case PXB_BC_RE_TRANSMISSIVE:
            add(0, t[0]);
            add(1, t[1]);
            add(2, t[2]);
            break;
        case PXB_BC_RE_TRANSMISSIVEBED:
        case PXB_BC_RE_STEEPFALL:
            add(3, t[3]);
            break;
        case PXB_BC_RE_NORMALFLOWDEPTH:  // hu, hv copied; h and z_b prescribed
            add(1, t[1]);
            add(2, t[2]);
            break;
        case PXB_BC_RE_ZEROMOMENTUM:  // NaN values keep the cell's own momentum (its donor)
            if (h.c0 != h.c0) add(1, t[1]);
            if (h.c1 != h.c1) add(2, t[2]);
            break;
        case PXB_BC_RE_CONSTANTINFLUX:  // prescribed hu = q values[1], hv = q values[2]: the adjoint of q
            if (h.qbar) {
                const double v = t[1] * h.vx + t[2] * h.vy;
                if (v != 0.0) atomicAdd(h.qbar, v);
            }
            break;
        default:  // Berthon: prescribed values
            break;
    }
}

// Handlers backwards, the last one first, by one block.  A thread keeps what it takes of a
// handler's cells, at most ADJ_BC_KEEP, in registers; the next handler's indices are read ahead.
// Bound by the chain of loads, barrier and atomics of each handler: 2.7 us for one of 514 cells,
// 4.5 for 1026 and 2048.  Beyond the registers one block pays for every 1024 cells more (4096
// cells 9 us, 65536 166 us); two launches over all cells take 3.7 to 5.5 us for any of them
// (three took 7).
constexpr int ADJ_BC_KEEP = 2;
static_assert(ADJ_BC_KEEP * 1024 == ADJ_BC_SET_CELLS, "a block of 1024 threads keeps a handler's cells");
__global__ void __launch_bounds__(1024) adj_bc_set_kernel(const __grid_constant__ AdjBcSet a) {
    const int nt = blockDim.x;
    long long cell[ADJ_BC_KEEP], donor[ADJ_BC_KEEP];
    auto ahead = [&](int q) {
#pragma unroll
        for (int u = 0; u < ADJ_BC_KEEP; ++u) {
            const int k = threadIdx.x + u * nt;
            cell[u] = donor[u] = 0;
            if (k < a.h[q].count) cell[u] = a.h[q].cells[k], donor[u] = a.h[q].donors[k];
        }
    };
    ahead(a.n - 1);
    for (int q = a.n - 1; q >= 0; --q) {
        const AdjBcHandler& h = a.h[q];
        double t[ADJ_BC_KEEP][6];
        long long d[ADJ_BC_KEEP];
#pragma unroll
        for (int u = 0; u < ADJ_BC_KEEP; ++u) {
            d[u] = donor[u];
            if ((int)threadIdx.x + u * nt < h.count) adj_bc_take(a, h, cell[u], t[u]);
        }
        if (q > 0) ahead(q - 1);
        __syncthreads();  // every clear before any addition
#pragma unroll
        for (int u = 0; u < ADJ_BC_KEEP; ++u)
            if ((int)threadIdx.x + u * nt < h.count) adj_bc_give(a, h, d[u], t[u]);
        if (q > 0) {
            __threadfence();
            __syncthreads();
        }
    }
}

// One handler of more cells (a.h[0]) in two launches over all of them: take, then give.
__global__ void __launch_bounds__(256) adj_bc_take_kernel(const __grid_constant__ AdjBcSet a) {
    const AdjBcHandler& h = a.h[0];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= h.count) return;
    double t[6];
    adj_bc_take(a, h, h.cells[k], t);
#pragma unroll
    for (int s = 0; s < 6; ++s) a.tmp[(size_t)s * h.count + k] = t[s];
}

__global__ void __launch_bounds__(256) adj_bc_give_kernel(const __grid_constant__ AdjBcSet a) {
    const AdjBcHandler& h = a.h[0];
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= h.count) return;
    double t[6];
#pragma unroll
    for (int s = 0; s < 6; ++s) t[s] = a.tmp[(size_t)s * h.count + k];
    adj_bc_give(a, h, h.donors[k], t);
}

// compute_n of the initialisation backwards (roe_exner.py:64-73): n_b = n_p_mix where the
// raw z_b > SED_TOL (MPM), the raw n elsewhere (and everywhere with a constant grass
// factor).  The n_b adjoint moves to n (when nbar is set) or to n_p_mix (summed into
// *npbar); n_b's own value before the initialisation has no influence.
__global__ void __launch_bounds__(256) adj_compute_n_kernel(int ny, int nx, long long pitch, int mpm,
                                                            const double* zb, double* nbbar, double* nbar,
                                                            double* npbar) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    double v[1] = {0.0};
    if (r < ny && c < nx) {
        const long long i = (long long)r * pitch + c;
        const double b = nbbar[i];
        if (mpm && zb[i] > SED_TOL) v[0] = b;
        else if (nbar) nbar[i] += b;
        nbbar[i] = 0.0;
    }
    adj_sum_add<1>(npbar, v);
}

// ---------------------------------------------------------------- dt backwards

__device__ __forceinline__ bool adj_face_speed(const AdjCflArgs& a, int r, int c, bool yf, double& s) {
    if (yf ? (r + 1 >= a.ny) : (c + 1 >= a.nx)) return false;
    const long long i = (long long)r * a.pitch + c, j = yf ? i + a.pitch : i + 1;
    if (!(((a.h[i] > DRY_TOL) || (a.h[j] > DRY_TOL)) && !(adj_nodata(a.nodata, i) || adj_nodata(a.nodata, j))))
        return false;
    const CCell<double> I = make_ccell(a.h[i], a.hu[i], a.hv[i], a.G[i]);
    const CCell<double> J = make_ccell(a.h[j], a.hu[j], a.hv[j], a.G[j]);
    s = yf ? face_speed<double, true>(I, J) : face_speed<double, false>(I, J);
    return true;
}

// Whether a face's speed is the maximum: its bound from the two cells rules most faces out
// (cfl_bound) before the speed itself is formed.
__device__ __forceinline__ bool adj_at_max(const AdjCflArgs& a, int r, int c, bool yf, unsigned long long m, float smax) {
    if (yf ? (r + 1 >= a.ny) : (c + 1 >= a.nx)) return false;
    const long long i = (long long)r * a.pitch + c, j = yf ? i + a.pitch : i + 1;
    const float hi = clamp_lo((float)a.h[i], (float)DRY_TOL), hj = clamp_lo((float)a.h[j], (float)DRY_TOL);
    const float ri = f_rcp(hi), rj = f_rcp(hj);
    const float U = fmax_nan(fabsf((float)a.hu[i]) * ri, fabsf((float)a.hu[j]) * rj);
    const float V = fmax_nan(fabsf((float)a.hv[i]) * ri, fabsf((float)a.hv[j]) * rj);
    const float b = cfl_bound(U, V, fmax_nan(hi, hj), fminf(hi, hj), fmax_nan(fabsf((float)a.G[i]), fabsf((float)a.G[j])));
    double s;
    return !(b < smax) && adj_face_speed(a, r, c, yf, s) && speed_bits(s) == m;
}

// pass 1: number of faces at the maximum speed
__global__ void __launch_bounds__(256) adj_cfl_ties_kernel(const AdjCflArgs a) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (r >= a.ny || c >= a.nx) return;
    const unsigned long long m = *a.maxbits;
    const float smax = (float)bits_speed(m, 0.0);
    unsigned int ties = 0;
    for (int yf = 0; yf < 2; ++yf) ties += adj_at_max(a, r, c, yf != 0, m, smax) ? 1u : 0u;
    if (ties) atomicAdd(a.nties, ties);
}

// pass 2: d(dt)/d(s_max) spread over the tying faces, through their speeds' local Jacobians
__global__ void __launch_bounds__(256) adj_cfl_grad_kernel(const AdjCflArgs a) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y * blockDim.y + threadIdx.y;
    if (r >= a.ny || c >= a.nx) return;
    const unsigned long long m = *a.maxbits;
    const double smax = bits_speed(m, 0.0);
    const double dt = a.cfl * (a.dx / smax);
    if (!(dt >= a.floor_dt) || *a.nties == 0u) return;  // the floor (or no face): dt does not depend on the state
    const double sbar = *a.dtbar * (-a.cfl * a.dx / (smax * smax)) / (double)*a.nties;
    for (int yf = 0; yf < 2; ++yf) {
        if (!adj_at_max(a, r, c, yf != 0, m, (float)smax)) continue;
        using D = DualN<8>;
        const long long i = (long long)r * a.pitch + c, j = yf ? i + a.pitch : i + 1;
        const CCell<D> I = make_ccell(D::seed(a.h[i], 0), D::seed(a.hu[i], 1), D::seed(a.hv[i], 2), D::seed(a.G[i], 3));
        const CCell<D> J = make_ccell(D::seed(a.h[j], 4), D::seed(a.hu[j], 5), D::seed(a.hv[j], 6), D::seed(a.G[j], 7));
        const D sd = yf ? face_speed<D, true>(I, J) : face_speed<D, false>(I, J);
        atomicAdd(a.Ah + i, sbar * sd.d[0]);
        atomicAdd(a.Ahu + i, sbar * sd.d[1]);
        atomicAdd(a.Ahv + i, sbar * sd.d[2]);
        atomicAdd(a.AG + i, sbar * sd.d[3]);
        atomicAdd(a.Ah + j, sbar * sd.d[4]);
        atomicAdd(a.Ahu + j, sbar * sd.d[5]);
        atomicAdd(a.Ahv + j, sbar * sd.d[6]);
        atomicAdd(a.AG + j, sbar * sd.d[7]);
    }
}

}  // namespace pxb
