// Launches of the several-steps-per-launch tile kernel (llb_tile.cuh) for every
// storage form.  Compiled with --fmad=false, like the other step kernels, so
// its arithmetic rounds as theirs.
#include "llb_tile.cuh"

#include <algorithm>
#include <type_traits>

#include "../../include/llalbm_cuda.h"
#include "llb_launch.h"
#include "llb_pdl.cuh"

namespace llb {

namespace {

template <class M, int CPW>
cudaError_t do_step_tile(const LaunchCtx& x, const TilePlan& p, const void* fin, void* fout, int steps, bool macro) {
    using T = typename M::T;
    const int V = 32 * Rows<M, 1>::RPL - 2 * p.H;
    const int RC = p.TJ + 2 * steps, nw = (RC + CPW - 1) / CPW;
    const dim3 grid((x.g.rows + V - 1) / V, (x.g.cols + p.TJ - 1) / p.TJ), block(32 * nw);
    const T* in = static_cast<const T*>(fin);
    T* out = static_cast<T*>(fout);
    const int smem = tile_smem_bytes(nw, CPW, x.g.ps != nullptr);
    auto kern = x.c.model == 0 ? k_step_tile<M, 0, CPW, false> : k_step_tile<M, 1, CPW, false>;
    if constexpr (std::is_same_v<M, ModelF64>)
        if (x.g.ps) kern = x.c.model == 0 ? k_step_tile<M, 0, CPW, true> : k_step_tile<M, 1, CPW, true>;
    // The limit belongs to the kernel, which every handle shares: the most any of
    // its launches takes, so that what another thread sets is the same.
    const int most = tile_smem_bytes(TILE_MAX_WARPS, CPW, x.g.ps != nullptr);
    if (most > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return e;
    }
    return launch_pdl_smem(kern, grid, block, smem, x.stream, x.g, x.ot, x.c, in, out, x.mo, x.ss, steps, p.H, p.TJ,
                           macro ? 1 : 0);
}

template <class M>
cudaError_t step_tile(const LaunchCtx& x, const TilePlan& p, const void* fin, void* fout, int steps, bool macro) {
    switch (p.CPW) {
    case 1: return do_step_tile<M, 1>(x, p, fin, fout, steps, macro);
    case 2: return do_step_tile<M, 2>(x, p, fin, fout, steps, macro);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// The shape whose launches cost least per step, among those with a tile per SM
// at most: a launch's fixed cost and the load of a tile, and per step the larger
// of one warp's chain over its columns and the columns a tile updates (0.05 us a
// column in every form: about 200 instructions on one of four schedulers).  The
// model ranks shapes and no more (129^2 FP64: 0.85 us by it, 1.5 measured); out
// of every shape measured on 31 lattices x forms it chose one within 9 % of the
// best and 1.2 % of it on average.
//
// With no more tiles than SMs every block starts at once.  With two or more per
// SM the second wave's launch ends long after the first's, and whether tiles win
// is chance: us a step, one-step kernels / tiles, FP64 256 x 400 4.40 / 4.68, TRT
// 4.43 / 5.14, 300 x 380 4.26 / 4.70, TRT 4.30 / 5.29, 3 x 30000 26.4 / 28.3;
// FP32 400 x 490 4.40 / 4.96, 16 x 12000 10.2 / 14.2; FP16 10 x 4000 6.9 / 9.0,
// 130 x 3000 8.9 / 9.9, 7 x 13053 11.5 / 25.2 (and some gain: FP64 16 x 7000
// 7.76 / 5.86, FP32 channel 400 x 490 4.62 / 4.20).
//
// One wave, us a step, one-step kernels / tiles: FP64 64^2 1.93 / 1.34, 129^2
// 3.22 / 1.52, 181 x 333 3.72 / 3.04, TRT 3.73 / 3.32, 1492 x 43 TRT 3.28 / 2.99;
// FP32 129^2 3.09 / 1.62, 256 x 400 3.97 / 3.02, 440 x 450 4.40 / 3.95; FP16 64^2
// 1.82 / 2.00 (the cluster kernel), 129^2 3.27 / 1.90, 256 x 1024 6.06 / 5.13,
// 680 x 578 6.92 / 5.94.  Two columns a warp are not taken with partially
// saturated obstacles (100 x 250, one column, 3.33 / 2.10; 200 x 249, two, 3.42 /
// 3.60, TRT 3.44 / 3.82) and not against the cluster kernel, whose lattices need
// them only when they are a few rows high, most of a tile outside (3 x 3900 FP64
// 2.1 / 4.1, FP32 1.9 / 5.0; 8 x 3000 FP16 1.17 times the cluster's).
//
// A launch costs its load and its halo however few steps it takes.  us a step,
// one-step kernels / tiles: launches of one step FP64 181 x 333 3.9 / 4.9, FP16
// 256 x 1024 6.4 / 8.3, FP64 129^2 3.4 / 3.2; of two, one column a warp, 129^2 3.4 /
// 2.1; two columns FP64 1492 x 43 3.4 / 3.6, TRT 3.4 / 3.8, FP16 256 x 1024 6.4 /
// 6.1; of three 3.4 / 3.1, TRT 3.4 / 3.35, 6.4 / 5.5.  So two steps at least, three
// with two columns.  In FP16 a lane writes the
// output of its four rows one after the other, 32 bytes apart across the warp,
// which with two columns costs more than the one-step kernel's output step: a
// run of two steps with output 256 x 1024 6.6 / 8.1, of three 6.5 / 7.0.
bool tile_plan(int storage, int R, int C, bool partial, bool cluster, int sm_count, TilePlan* plan) {
    *plan = TilePlan{};
    const int form = partial ? 3 : storage == LLB_STORE_F64 ? 0 : storage == LLB_STORE_F32S ? 1 : 2;
    static constexpr long long kMost[4] = {115000, 200000, 400000, 50000}, kLeast[4] = {0, 0, 8000, 0};
    const long long nodes = static_cast<long long>(R) * C;
    if (nodes > kMost[form] || nodes < kLeast[form]) return false;
    const int rpl = form == 1 ? 2 : form == 2 ? 4 : 1;
    const int most_cpw = partial || cluster ? 1 : 2;
    double best = 1e30;
    for (int T : {3, 4, 5, 6, 8})
        for (int cpw = 1; cpw <= most_cpw; ++cpw)
            for (int nw = 8; nw <= 16; nw += 2) {
                const int H = (T + rpl - 1) / rpl * rpl, V = 32 * rpl - 2 * H, TJ = nw * cpw - 2 * T;
                if (TJ < 2) continue;
                const long long tiles = static_cast<long long>((R + V - 1) / V) * ((C + TJ - 1) / TJ);
                if (tiles > sm_count) continue;
                const double step = std::max(0.1 + 0.4 * cpw, 0.05 * (nw * cpw - T));
                const double t = (1.5 + T * step) / T;
                if (t < best) {
                    best = t;
                    *plan = TilePlan{T, H, TJ, cpw, cpw == 2 ? 3 : 2, form == 2 && cpw == 2};
                }
            }
    return plan->T > 0;
}

cudaError_t launch_step_tile(int storage, const LaunchCtx& x, const TilePlan& p, const void* fin, void* fout,
                             int steps, bool macro) {
    switch (storage) {
    case LLB_STORE_F64: return step_tile<ModelF64>(x, p, fin, fout, steps, macro);
    case LLB_STORE_F32S: return step_tile<ModelShift<float>>(x, p, fin, fout, steps, macro);
    default: return step_tile<ModelShift<__half>>(x, p, fin, fout, steps, macro);
    }
}

}  // namespace llb
