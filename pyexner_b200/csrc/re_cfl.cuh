// CFL reduction for the Roe-Exner bundle (compute_dt_roeexner,
// PyExner src/PyExner/solvers/roe_exner_solver.py:118-122 with compute_dt_2D,
// roe_exner.py:257-310).
//
// min over active faces of dx / speed_f equals dx / max_f speed_f exactly (division by
// a positive number is monotone under round-to-nearest), so the kernel reduces the
// maximum speed: a warp-level max of the IEEE bit patterns (speeds are >= 0 or NaN, so
// unsigned order is float order and NaN wins like jnp.min's NaN), a block max through
// shared memory, one 64-bit atomicMax per block, and the last block to finish turns it
// into dt = max(cfl * dx / smax, 1e-6),
// resets the accumulator and logs dt.  Deterministic and free of host round trips.
//
// Work layout: a warp takes an item, a strip of a band of rows.  Narrow items (small grids)
// evaluate every face of 31 columns.  Wide items (124 columns, four per lane) read every
// cell once, 16 bytes per lane and plane, and form for each row an upper bound of the speeds
// of its faces: the largest over the lanes, each from the extremes of h, |u|, |v| and G
// among the ten cells its faces join.  Exact speeds of one row of 31 columns per item,
// spread over the grid, give a lower bound of the maximum; only rows whose bound is not
// below what is known by then are evaluated face by face, as narrow items of up to four rows
// shared out over the block's warps (they lie close together: left to the warp that found
// them, one warp's rows set the kernel's time).  A face that is left out cannot be the
// fastest, so dt keeps its bits.
//
// Bound by the read of h, hu, hv and G (8192^2: 5.9 TB/s) and, on small grids, by the chain
// of launch, loads, reduction and last block.  Evaluating every face takes 125 to 300
// instructions per row of 31.  us with every face evaluated (by 16-byte row copies in
// float32) -> now: float32 514^2 8.1 -> 5.9 and with a constant G 11.1 -> 7.6; 2050^2 24.5 ->
// 15.6 below the bedload threshold, 53 -> 25 with bedload or a constant G everywhere; 4098^2
// 82 -> 55 and 192 -> 70; float64 1026^2 27 -> 17 and 77 -> 52; 2050^2 93 -> 36 and 284 -> 95.
// In a field whose cells differ from one another like noise no row is ruled out and every
// face is evaluated after the bounds: float32 2050^2 256 -> 225, float64 1026^2 70 -> 92,
// 2050^2 263 -> 339.
#pragma once
#include <algorithm>
#include <type_traits>

#include "pxb_device.cuh"

namespace pxb {

struct CflScratch {
    unsigned long long maxbits;  // running max of speed bits
    unsigned long long last;     // the largest speed of the last completed reduction (bits)
    unsigned int done;           // finished blocks of the current launch
    unsigned int step;           // index into the dt log
    int err;                     // sticky error word
    int pad;
    double t_step;               // simulation time at the start of the current step
    double t_next;               // t_step + dt: the time the next dt is added to
};

// Start of a fixed-step run at time t0 (the first CFL launch moves it into t_step).
template <class T>
__global__ void set_time_kernel(CflScratch* scr, double t0) {
    scr->t_step = t0;
    scr->t_next = t0;
}

template <class T>
struct CflArgs {
    int ny, nx;
    long long pitch;
    const T *h, *hu, *hv, *G;
    const uint8_t* nodata;
    T dx, cfl, floor_dt;  // floor_dt = 1e-6 (Roe-Exner); <= 0 disables the floor
    CflScratch* scr;
    T* dt_out;   // device scalar
    T* dt_log;   // optional: dt_log[scr->step++] = dt
    int band_rows, nstrips, nbands;
    int wide;  // items are 124 columns wide with bounds (else 31, every face)
};

constexpr int CFL_WIDE = 124, CFL_NARROW = 31;  // columns of an item
constexpr int CFL_MAX_ROWS = 64;                // rows of a wide item (a lane keeps two bounds)
constexpr int CFL_CHUNK = 4;  // rows of an item that are evaluated together (4096^2 at rest, float32: 58 us with 16, 55 with 4)
static_assert(CFL_WIDE % CFL_NARROW == 0 && 32 % CFL_CHUNK == 0, "shapes of the wide items");

// Work items of the reduction over a grid, 8 a block.
struct CflItems {
    int band_rows = 0, nstrips = 0, nbands = 0, grid = 0;
    bool wide = false;
};
// Items of one width, about 32 warps of them per SM (16: 24 to 30 % slower at 2048^2, 64 as
// well).
static inline CflItems cfl_items(int ny, int nx, bool wide, int sm_count) {
    CflItems g;
    g.wide = wide;
    g.nstrips = wide ? (nx + CFL_WIDE - 1) / CFL_WIDE : (nx + CFL_NARROW - 1) / CFL_NARROW;
    const int want = std::max(1, 32 * sm_count / g.nstrips);
    g.band_rows = std::max(2, (ny + want - 1) / want);
    if (wide) g.band_rows = std::min(CFL_MAX_ROWS, std::max(4, g.band_rows));
    g.nbands = (ny + g.band_rows - 1) / g.band_rows;
    g.grid = (int)(((long long)g.nstrips * g.nbands + 7) / 8);
    return g;
}
// A plan's items.  Below the line a wide item's bounds cost more than evaluating every face of
// narrow items.  us narrow / wide, at rest and with bedload everywhere: float32 770^2 7.1 / 9.5
// and 11.9 / 13.0, 1026^2 8.5 / 10.0 and 16.3 / 14.8, 1400^2 11.5 / 13.7 and 25.2 / 17.9, 2050^2
// 19.5 / 15.8 and 47.9 / 25.6; float64 640^2 15.8 / 15.1 and 37.6 / 82, 770^2 21.1 / 16.5 and
// 56.8 / 44.8, 1026^2 31 / 17 and 87 / 50, 2050^2 115 / 36 and 305 / 93.
static inline CflItems cfl_items(int ny, int nx, int esize, int sm_count) {
    return cfl_items(ny, nx, (long long)ny * nx > (esize == 8 ? 500000 : 1200000), sm_count);
}

// Resident 256-thread blocks per SM: 4 (64 registers; the spills are in the exact rows of wide
// items) against 2 and 3 is 15 to 30 % faster at 8192^2 in float32.
constexpr int cfl_min_blocks(int esize) { return esize == 8 ? 2 : 4; }

template <class T>
using speed_bits_t = typename std::conditional<sizeof(T) == 4, unsigned, unsigned long long>::type;

__device__ __forceinline__ unsigned warp_max_bits(unsigned v) { return __reduce_max_sync(FULL, v); }
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(FULL, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// The x-faces (c | c+1) of rows r0 .. r1-1 and the y-faces (r | r+1) below them, for the 31
// columns from c0 (the 32nd lane is the east neighbour of the last).
template <class T, bool HAS_MASK>
__device__ __forceinline__ void cfl_rows(const CflArgs<T>& a, const int c0, const int r0, const int r1,
                                         speed_bits_t<T>& best) {
    const int lane = threadIdx.x & 31;
    const int ny = a.ny, nx = a.nx, c = c0 + lane;
    const bool colok = c < nx, has_e = lane < 31 && c + 1 < nx;
    const T DRY = T(DRY_TOL);
    struct Raw { T h, hu, hv, g; bool m; };
    auto load = [&](int r) __attribute__((always_inline)) {
        Raw x{T(1), T(0), T(0), T(0), false};
        if (colok && r < ny) {
            const long long i = (long long)r * a.pitch + c;
            x.h = __ldg(a.h + i);
            x.hu = __ldg(a.hu + i);
            x.hv = __ldg(a.hv + i);
            x.g = __ldg(a.G + i);
            if (HAS_MASK) x.m = __ldg(a.nodata + i) != 0;
        }
        return x;
    };
    auto fold = [&](bool act, T s) __attribute__((always_inline)) {
        const speed_bits_t<T> b = (speed_bits_t<T>)speed_bits(s);
        best = act && b > best ? b : best;
    };
    Raw x = load(r0), nx_ = load(r0 + 1);
    CCell<T> cur = make_ccell(x.h, x.hu, x.hv, x.g);
    bool m = x.m;
    for (int r = r0; r < r1; ++r) {
        const CCell<T> s = make_ccell(nx_.h, nx_.hu, nx_.hv, nx_.g);
        const bool ms = nx_.m;
        if (r + 1 < r1) nx_ = load(r + 2);  // in flight during this row's faces
        // rows r and r+1 without G (below the Shields threshold) take face_speed_nog, the
        // same value without a~ and the cubic (a NaN G is not 0)
        const bool nog = !__any_sync(FULL, !(cur.G == T(0)) || !(s.G == T(0)));
        CCell<T> e;
        e.h = __shfl_down_sync(FULL, cur.h, 1);
        e.sq = __shfl_down_sync(FULL, cur.sq, 1);
        e.u = __shfl_down_sync(FULL, cur.u, 1);
        e.v = __shfl_down_sync(FULL, cur.v, 1);
        const bool me = HAS_MASK ? (__shfl_down_sync(FULL, (int)m, 1) != 0) : false;
        // cur.h = max(h, DRY_TOL) > DRY_TOL exactly when h > DRY_TOL (false for NaN)
        const bool ax = has_e && ((cur.h > DRY) || (e.h > DRY)) && !(m || me);
        const bool ay = colok && r + 1 < ny && ((cur.h > DRY) || (s.h > DRY)) && !(m || ms);
        if (nog) {
            fold(ax, face_speed_nog<T, false>(cur, e));
            fold(ay, face_speed_nog<T, true>(cur, s));
        } else {
            e.G = __shfl_down_sync(FULL, cur.G, 1);
            e.rs = __shfl_down_sync(FULL, cur.rs, 1);
            // only active faces enter the cubic: a lane without a face could otherwise send
            // the whole warp into the float64 fallback of the float32 solve
            if (ax) fold(true, face_speed<T, false>(cur, e));
            if (ay) fold(true, face_speed<T, true>(cur, s));
        }
        cur = s;
        m = ms;
    }
}

// max / min that propagate NaN (max only: a NaN minimum goes with a NaN maximum)
__device__ __forceinline__ float fmax_nan(float a, float b) { float y; asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b)); return y; }

// Upper bound of the face speeds among cells with depths (clamped at DRY_TOL) in [hm, hM],
// velocity components up to U and V and grass factors up to G, with a margin for the rounding
// of the bound and of the speeds.  With M the larger of U and V and m the other, a face's
// normal velocities and u~ are up to M and its c~ lies between the cells' sqrt(g h).  Without
// G the speeds are |u~| + c~.  With G they are the roots of
//   l ((l - u)^2 - c^2) = a c^2 (l + u),  a <= A = G (3 M^2 + m^2) / hm
// (the sign of l turned; u >= 0).  A positive root has l <= u - c, or l >= u + c and then
// (l - u)^2 = c^2 (1 + a (1 + u / l)) with u / l <= u / (u + c) <= M / (M + cm); a negative
// one has |l| <= c sqrt(1 + a) - u.  The trigonometric solution gives the roots when all three
// are real; at l = -(c - u)/2 the left side less the right is at least
// (c - u)^2 (3 c + u) / 8 - a c^2 u, which is positive, and all three are, when
// A cM^2 M < 0.375 (cm - M)^2 cm.  Otherwise its argument is clipped and its values are
// within 4/3 |u| + 2/sqrt(3) c sqrt(1 + a).  A NaN makes the bound NaN.
__device__ __forceinline__ float cfl_bound(float U, float V, float hM, float hm, float G) {
    const float cM = f_sqrt(9.81f * hM), M = fmax_nan(U, V);
    if (G == 0.f) return (M + cM) * 1.00002f;
    const float m = fminf(U, V), cs = f_sqrt(9.81f * hm), cm = cs - M;
    const float A = G * (3.f * M * M + m * m) / hm * 1.0001f;
    const bool three = cm > 0.f && A * cM * cM * M < 0.374f * cm * cm * cs;
    const float tight = M + cM * f_sqrt(1.f + A * (1.f + M * f_rcp(M + cs)));
    const float loose = 1.3334f * M + 1.1548f * cM * f_sqrt(1.f + A);
    return (three ? tight : loose) * 1.0002f;
}

// A wide item: strip, rows, and this lane's four columns.
template <class T>
struct CflStrip {
    int c, R0, R1;  // this lane's first column (lane 31: the next strip's), rows
    bool inner;     // every column of the strip lies in the grid
    __device__ __forceinline__ CflStrip(const CflArgs<T>& a, int item) {
        const int band = item / a.nstrips, c0 = (item - band * a.nstrips) * CFL_WIDE;
        c = c0 + 4 * (threadIdx.x & 31);
        R0 = band * a.band_rows;
        R1 = min(a.ny, R0 + a.band_rows);
        inner = c0 + 128 <= a.nx;
    }
};
template <class T>
struct CflRow {
    T h[4], hu[4], hv[4], g[4];
};

template <class T>
__device__ __forceinline__ void cfl_load4(const T* p, T (&v)[4]) {
    if constexpr (sizeof(T) == 4) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    } else {
        const double2 t = __ldg(reinterpret_cast<const double2*>(p)), w = __ldg(reinterpret_cast<const double2*>(p) + 1);
        v[0] = t.x, v[1] = t.y, v[2] = w.x, v[3] = w.y;
    }
}

// Row r of a lane's four columns.  VEC: 16-byte aligned planes and a pitch of whole groups
// of four elements; a group that reaches beyond the grid is loaded element by element (a
// plane ends with its last cell).  Columns beyond the grid: still water of no depth, without G.
template <class T, bool VEC>
__device__ __forceinline__ void cfl_load(const CflArgs<T>& a, const CflStrip<T>& st, int r, CflRow<T>& x) {
    const long long i = (long long)r * a.pitch + st.c;
    if (VEC && (st.inner || st.c + 4 <= a.nx)) {
        cfl_load4(a.h + i, x.h);
        cfl_load4(a.hu + i, x.hu);
        cfl_load4(a.hv + i, x.hv);
        cfl_load4(a.G + i, x.g);
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool ok = st.c + k < a.nx;
            x.h[k] = ok ? __ldg(a.h + i + k) : T(0);
            x.hu[k] = ok ? __ldg(a.hu + i + k) : T(0);
            x.hv[k] = ok ? __ldg(a.hv + i + k) : T(0);
            x.g[k] = ok ? __ldg(a.G + i + k) : T(0);
        }
    }
}

// Bounds of the rows of a wide item (x-faces of row r, y-faces (r | r+1)): lane k gets those
// of rows R0 + k and R0 + 32 + k.
template <class T, bool VEC>
__device__ __forceinline__ void cfl_wide_bounds(const CflArgs<T>& a, const CflStrip<T>& st, float& bound0, float& bound1) {
    const int lane = threadIdx.x & 31, R0 = st.R0, R1 = st.R1, rend = min(a.ny, R1 + 1);
    using Row = CflRow<T>;
    auto load = [&](int r, Row& x) __attribute__((always_inline)) { cfl_load<T, VEC>(a, st, r, x); };
    // extremes of this lane's four cells of a row and the next column's
    struct Ext { float U, V, hM, hm, G; };
    auto extremes = [&](const Row& x) __attribute__((always_inline)) {
        Ext e{0.f, 0.f, 0.f, 3e38f, 0.f};
        float h0 = 0.f, u0 = 0.f, v0 = 0.f, g = 0.f, g0 = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float h = clamp_lo((float)x.h[k], (float)DRY_TOL), r = f_rcp(h);
            const float u = fabsf((float)x.hu[k]) * r, v = fabsf((float)x.hv[k]) * r;
            if (k == 0) h0 = h, u0 = u, v0 = v;
            e.U = fmax_nan(e.U, u);
            e.V = fmax_nan(e.V, v);
            e.hM = fmax_nan(e.hM, h);
            e.hm = fminf(e.hm, h);
            g = fmax_nan(g, fabsf((float)x.g[k]));
            if (k == 0) g0 = g;
        }
        e.G = fmax_nan(g, __shfl_down_sync(FULL, g0, 1));
        const float he = __shfl_down_sync(FULL, h0, 1);
        e.U = fmax_nan(e.U, __shfl_down_sync(FULL, u0, 1));
        e.V = fmax_nan(e.V, __shfl_down_sync(FULL, v0, 1));
        e.hM = fmax_nan(e.hM, he);
        e.hm = fminf(e.hm, he);
        return e;
    };
    Row cur, nxt;
    load(R0, cur);
    if (R0 + 1 < rend) load(R0 + 1, nxt);
    Ext pe = extremes(cur);
    for (int r = R0; r < R1; ++r) {
        Ext ce = pe;
        if (r + 1 < rend) {
            cur = nxt;
            if (r + 2 < rend) load(r + 2, nxt);
            ce = extremes(cur);
        }
        const float b = cfl_bound(fmax_nan(pe.U, ce.U), fmax_nan(pe.V, ce.V), fmax_nan(pe.hM, ce.hM), fminf(pe.hm, ce.hm),
                                  fmax_nan(pe.G, ce.G));
        const float w = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(b)));  // (NaN above all numbers)
        const int k = r - R0;
        if (lane == (k & 31)) (k < 32 ? bound0 : bound1) = w;
        pe = ce;
    }
}

// Rows left to evaluate by a block of 8 warps, in chunks of CFL_CHUNK rows of an item.
struct CflTasks {
    int count;
    float bound[8 * CFL_MAX_ROWS / CFL_CHUNK];
    unsigned char warp[8 * CFL_MAX_ROWS / CFL_CHUNK], first[8 * CFL_MAX_ROWS / CFL_CHUNK], last[8 * CFL_MAX_ROWS / CFL_CHUNK];
};

// Wide items of a block, one per warp (`item`: this warp's, negative for none; `items`: all
// warps').  Every warp forms its rows' bounds; the rows that
// may hold the maximum, which tend to lie in few items, are shared out over the block: a warp
// evaluates every face of 31 columns of a chunk's rows, as a narrow item.
// Returns with the maximum covering whatever the block's warps could not rule out.
template <class T, bool HAS_MASK, bool VEC>
__device__ __forceinline__ void cfl_wide_block(const CflArgs<T>& a, const int item, const int* items, CflTasks& tasks) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long seen = 0ull;  // the maximum as last read, in lane 0
    if (threadIdx.x == 0) tasks.count = 0;
    __syncthreads();
    if (item >= 0) {
        const CflStrip<T> st(a, item);
        speed_bits_t<T> best = 0;
        {  // the faces of a row of 31 columns somewhere in the grid: items in order step through
           // the rows, and through the columns by the golden ratio
            const int r = (int)((long long)a.ny * item / (a.nstrips * a.nbands));
            const int cs = (int)(((unsigned)item * 2654435769u >> 8) * (unsigned long long)max(1, a.nx - 31) >> 24);
            cfl_rows<T, HAS_MASK>(a, cs, r, r + 1, best);
            best = warp_max_bits(best);
            if (lane == 0 && best) atomicMax(&a.scr->maxbits, (unsigned long long)best);
        }
        float b0 = 0.f, b1 = 0.f;
        cfl_wide_bounds<T, VEC>(a, st, b0, b1);
        if (lane == 0) seen = *(volatile unsigned long long*)&a.scr->maxbits;
        const float known = (float)bits_speed(__shfl_sync(FULL, seen, 0), T(0));
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float b = n ? b1 : b0;
            const bool todo = !(b < known) && st.R0 + 32 * n + lane < st.R1;  // (a NaN bound is not below it)
            const unsigned vote = __ballot_sync(FULL, todo);
            for (int k = 0; k < 32; k += CFL_CHUNK) {
                const unsigned bits = vote >> k & ((1u << CFL_CHUNK) - 1u);
                if (bits == 0u) continue;
                const bool mine = todo && lane >= k && lane < k + CFL_CHUNK;
                const unsigned most = __reduce_max_sync(FULL, mine ? __float_as_uint(b) : 0u);
                if (lane == 0) {
                    const int at = atomicAdd(&tasks.count, 1);
                    tasks.bound[at] = __uint_as_float(most);
                    tasks.warp[at] = (unsigned char)warp;
                    tasks.first[at] = (unsigned char)(32 * n + k + __ffs(bits) - 1);
                    tasks.last[at] = (unsigned char)(32 * n + k + 31 - __clz(bits));
                }
            }
        }
    }
    __syncthreads();
    constexpr int PARTS = CFL_WIDE / CFL_NARROW;
    for (int t = warp; t < PARTS * tasks.count; t += 8) {
        const int q = t / PARTS, part = t - PARTS * q;
        seen = __shfl_sync(FULL, seen, 0);
        if (tasks.bound[q] < (float)bits_speed(seen, T(0))) continue;
        const CflStrip<T> st(a, items[tasks.warp[q]]);
        const int c = st.c - 4 * lane + CFL_NARROW * part;
        if (c >= a.nx) continue;
        // (the maximum for the next chunk's test, in flight during this one)
        unsigned long long next = 0ull;
        if (lane == 0) next = *(volatile unsigned long long*)&a.scr->maxbits;
        speed_bits_t<T> best = 0;
        cfl_rows<T, HAS_MASK>(a, c, st.R0 + tasks.first[q], st.R0 + tasks.last[q] + 1, best);
        best = warp_max_bits(best);
        if (lane == 0 && (unsigned long long)best > seen) atomicMax(&a.scr->maxbits, (unsigned long long)best);
        seen = next;
    }
}

template <class T>
__device__ __forceinline__ bool cfl_aligned(const CflArgs<T>& a) {
    return ((((uintptr_t)a.h | (uintptr_t)a.hu | (uintptr_t)a.hv | (uintptr_t)a.G) & 15u) == 0) && ((a.pitch & 3) == 0);
}

// A narrow item: every face of 31 columns of a band, for this lane.
template <class T, bool HAS_MASK>
__device__ __forceinline__ void re_cfl_item(const CflArgs<T>& a, const int item, unsigned long long& best) {
    speed_bits_t<T> b = 0;
    const int band = item / a.nstrips, strip = item - band * a.nstrips;
    const int R0 = band * a.band_rows;
    cfl_rows<T, HAS_MASK>(a, strip * CFL_NARROW, R0, min(a.ny, R0 + a.band_rows), b);
    best = (unsigned long long)b > best ? (unsigned long long)b : best;
}

// One item per warp.  Wide items of one block lie far apart (the block number runs fastest),
// so that rows near the fastest faces end up in many blocks.
template <class T, bool HAS_MASK>
__global__ void __launch_bounds__(256, cfl_min_blocks(sizeof(T))) re_cfl_kernel(const __grid_constant__ CflArgs<T> a) {
    const int lane = threadIdx.x & 31;
    const int nitems = a.nstrips * a.nbands;
    unsigned long long best = 0ull;
    if (a.wide) {
        __shared__ CflTasks tasks;
        __shared__ int items[8];
        const int w = threadIdx.x >> 5, n = w * gridDim.x + blockIdx.x;
        const int item = n < nitems ? n : -1;
        if (lane == 0) items[w] = item;
        if (cfl_aligned(a)) cfl_wide_block<T, HAS_MASK, true>(a, item, items, tasks);
        else cfl_wide_block<T, HAS_MASK, false>(a, item, items, tasks);
        __syncthreads();  // the block's maxima before its ticket
    } else {
        const int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        if (item < nitems) re_cfl_item<T, HAS_MASK>(a, item, best);
    }
    // warp max, block max through shared memory, one atomic and one fence per block
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(FULL, best, o);
        best = other > best ? other : best;
    }
    __shared__ unsigned long long wmax[8];
    if (lane == 0) wmax[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int w = 1; w < 8; ++w) best = wmax[w] > best ? wmax[w] : best;
    if (best != 0ull) atomicMax(&a.scr->maxbits, best);
    __threadfence();  // the block's maximum before its ticket
    // last block finalises
    const unsigned int ticket = atomicAdd(&a.scr->done, 1u);
    if (ticket == gridDim.x - 1) {
        __threadfence();
        const unsigned long long bits = atomicAdd(&a.scr->maxbits, 0ull);
        const T smax = bits_speed(bits, T(0));
        // min_f dx/speed_f (inf when no face is active), then cfl * dt and the floor
        T dt = a.cfl * (a.dx / smax);
        if (a.floor_dt > T(0)) dt = clamp_lo(dt, a.floor_dt);
        *a.dt_out = dt;
        if (a.dt_log) a.dt_log[a.scr->step] = dt;
        a.scr->step += 1;
        // time of this step, accumulated in float64 like the host loops of the integrators
        a.scr->t_step = a.scr->t_next;
        a.scr->t_next = a.scr->t_next + (double)dt;
        if (!d_isfinite(dt)) a.scr->err |= 2;
        a.scr->last = bits;
        a.scr->maxbits = 0ull;
        a.scr->done = 0u;
        __threadfence();
    }
}

}  // namespace pxb
