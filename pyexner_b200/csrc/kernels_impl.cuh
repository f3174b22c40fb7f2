// Launchers shared by the float and double translation units.
#pragma once
#include <algorithm>
#include <type_traits>

#include "pxb_launch.h"

namespace pxb {

// Calls f with the compile-time flags (MPM, mask, averaged) of a stage kernel.
template <class F>
static cudaError_t stage_dispatch(bool mpm, bool hm, bool avg, F f) {
    using std::false_type;
    using std::true_type;
    switch ((mpm ? 4 : 0) | (hm ? 2 : 0) | (avg ? 1 : 0)) {
        case 0: return f(false_type{}, false_type{}, false_type{});
        case 1: return f(false_type{}, false_type{}, true_type{});
        case 2: return f(false_type{}, true_type{}, false_type{});
        case 3: return f(false_type{}, true_type{}, true_type{});
        case 4: return f(true_type{}, false_type{}, false_type{});
        case 5: return f(true_type{}, false_type{}, true_type{});
        case 6: return f(true_type{}, true_type{}, false_type{});
        default: return f(true_type{}, true_type{}, true_type{});
    }
}

template <class T>
cudaError_t launch_re_stage(const REStageArgs<T>& a, bool mpm, bool hm, bool avg, int grid, int threads, size_t smem,
                            cudaStream_t s) {
    return stage_dispatch(mpm, hm, avg, [&](auto M, auto H, auto A) {
        constexpr bool m = decltype(M)::value, h = decltype(H)::value, v = decltype(A)::value;
        // the budget variant only when its partial array is set (the others carry no budget code)
        if (a.bud) re_stage_kernel<T, m, h, v, true><<<grid, threads, smem, s>>>(a);
        else re_stage_kernel<T, m, h, v, false><<<grid, threads, smem, s>>>(a);
        return cudaGetLastError();
    });
}

template <class T>
cudaError_t launch_ens_stage(const EnsStageArgs<T>& a, bool mpm, bool hm, bool avg, int grid, int threads, size_t smem,
                             cudaStream_t s) {
    return stage_dispatch(mpm, hm, avg, [&](auto M, auto H, auto A) {
        constexpr bool m = decltype(M)::value, h = decltype(H)::value, v = decltype(A)::value;
        ens_stage_kernel<T, m, h, v><<<grid, threads, smem, s>>>(a);
        return cudaGetLastError();
    });
}

template <class T>
cudaError_t stage_allow_smem(bool mpm, bool hm, StageUse use, size_t bytes) {
    cudaError_t e = cudaSuccess;
    for (int avg = 0; avg < 2 && e == cudaSuccess; ++avg)
        e = stage_dispatch(mpm, hm, avg != 0, [&](auto M, auto H, auto A) {
            constexpr bool m = decltype(M)::value, h = decltype(H)::value, v = decltype(A)::value;
            const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
            if (use == STAGE_PLAN) return cudaFuncSetAttribute(re_stage_kernel<T, m, h, v, false>, at, (int)bytes);
            if (use == STAGE_BUDGET) return cudaFuncSetAttribute(re_stage_kernel<T, m, h, v, true>, at, (int)bytes);
            return cudaFuncSetAttribute(ens_stage_kernel<T, m, h, v>, at, (int)bytes);
        });
    return e;
}

template <class T>
cudaError_t launch_re_cfl(const CflArgs<T>& a, bool hm, int grid, cudaStream_t s) {
    if (hm) re_cfl_kernel<T, true><<<grid, 256, 0, s>>>(a);
    else re_cfl_kernel<T, false><<<grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_re_init(const InitArgs<T>& a, cudaStream_t s) {
    dim3 b(32, 8), g((a.nx + 31) / 32, (a.ny + 7) / 8);
    re_init_kernel<T><<<g, b, 0, s>>>(a);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_bc(const BcArgs<T>& a, cudaStream_t s) {
    if (a.h.count <= 0) return cudaSuccess;
    const int g = (a.h.count + 255) / 256;
    bc_gather_kernel<T><<<g, 256, 0, s>>>(a);
    bc_scatter_kernel<T><<<g, 256, 0, s>>>(a);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_bc_set(const BcSet<T>& a, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    // a warp for every 32 cells of a handler of the largest level (at most BC_SET_CHUNKS: the
    // host splits larger layouts), in the fewest blocks
    int most = 1, level = 0;
    for (int k = 0; k < a.n; ++k) {
        level = (a.h[k].level ? 0 : level) + (a.h[k].count + 31) / 32;
        most = std::max(most, level);
    }
    int blocks = 1;
    while (most > blocks * (BC_SET_THREADS / 32)) blocks *= 2;
    if (blocks > BC_SET_BLOCKS) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(32 * ((most + blocks - 1) / blocks));
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, bc_set_kernel<T>, a);
}

template <class T>
cudaError_t launch_ens_cfl(const EnsCflArgs<T>& a, bool hm, int grid, cudaStream_t s) {
    if (hm) ens_cfl_kernel<T, true><<<grid, 256, 0, s>>>(a);
    else ens_cfl_kernel<T, false><<<grid, 256, 0, s>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ens_cfl_finalize_kernel<T><<<(a.nmembers + 127) / 128, 128, 0, s>>>(a);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_re_general(const GenArgs<T>& a, int phase, cudaStream_t s) {
    dim3 b(32, 8), g((a.nx + 31) / 32, (a.ny + 7) / 8);
    switch (phase) {
        case GEN_HYDRO: gen_hydro_kernel<T><<<g, b, 0, s>>>(a); break;
        case GEN_CORR: gen_corr_kernel<T><<<g, b, 0, s>>>(a); break;
        case GEN_GRASS: gen_grass_kernel<T><<<g, b, 0, s>>>(a); break;
        case GEN_EXNER: gen_exner_kernel<T><<<g, b, 0, s>>>(a); break;
        default: gen_store_kernel<T><<<g, b, 0, s>>>(a); break;
    }
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_set_time(CflScratch* scr, double t0, cudaStream_t s) {
    set_time_kernel<T><<<1, 1, 0, s>>>(scr, t0);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_roe_stage(const RoeArgs<T>& a, bool avg, cudaStream_t s) {
    const int g = roe_tiles(a.nx, ROE_TX) * roe_tiles(a.ny, ROE_TY);
    if (avg) roe_stage_kernel<T, true><<<g, ROE_THREADS, 0, s>>>(a);
    else roe_stage_kernel<T, false><<<g, ROE_THREADS, 0, s>>>(a);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_budget_stage(const double* part, int nitems, const T* dt, double w_dx, BudgetAcc* acc,
                                cudaStream_t s) {
    budget_stage_kernel<T><<<1, 256, 0, s>>>(part, nitems, dt, w_dx, acc);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_volume(int ny, int nx, long long pitch, const T* h, const T* zb, const uint8_t* nodata,
                          double* part, int nblocks, double dx2, double* out, cudaStream_t s) {
    volume_kernel<T><<<nblocks, 256, 0, s>>>(ny, nx, pitch, h, zb, nodata, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    volume_final_kernel<<<1, 32, 0, s>>>(part, nblocks, dx2, out);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_roe_cfl(const CflArgs<T>& a, int grid, cudaStream_t s) {
    roe_cfl_kernel<T><<<grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

#define PXB_INSTANTIATE(T)                                                                              \
    template cudaError_t launch_re_stage<T>(const REStageArgs<T>&, bool, bool, bool, int, int, size_t, cudaStream_t); \
    template cudaError_t stage_allow_smem<T>(bool, bool, StageUse, size_t);                             \
    template cudaError_t launch_re_cfl<T>(const CflArgs<T>&, bool, int, cudaStream_t);                  \
    template cudaError_t launch_re_init<T>(const InitArgs<T>&, cudaStream_t);                           \
    template cudaError_t launch_bc<T>(const BcArgs<T>&, cudaStream_t);                                  \
    template cudaError_t launch_bc_set<T>(const BcSet<T>&, cudaStream_t);                               \
    template cudaError_t launch_re_general<T>(const GenArgs<T>&, int, cudaStream_t);                    \
    template cudaError_t launch_ens_stage<T>(const EnsStageArgs<T>&, bool, bool, bool, int, int, size_t, \
                                             cudaStream_t);                                             \
    template cudaError_t launch_ens_cfl<T>(const EnsCflArgs<T>&, bool, int, cudaStream_t);              \
    template cudaError_t launch_set_time<T>(CflScratch*, double, cudaStream_t);                         \
    template cudaError_t launch_roe_stage<T>(const RoeArgs<T>&, bool, cudaStream_t);                    \
    template cudaError_t launch_roe_cfl<T>(const CflArgs<T>&, int, cudaStream_t);                      \
    template cudaError_t launch_budget_stage<T>(const double*, int, const T*, double, BudgetAcc*, cudaStream_t); \
    template cudaError_t launch_volume<T>(int, int, long long, const T*, const T*, const uint8_t*, double*, int, \
                                          double, double*, cudaStream_t);

}  // namespace pxb
