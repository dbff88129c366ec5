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

// The shape whose launches cost least per step: a launch's fixed cost, the load
// of a tile, and per step the larger of one warp's chain over its columns and
// the columns an SM updates (0.05 us a column in every form: about 200
// instructions on one of four schedulers).  The model chose, out of every
// shape measured on 31 lattices x forms (40^2 to 500 x 800), one within 9 % of
// the best and 1.2 % of it on average.
//
// Lattices in the range below gain; us a step on B200, default kernel before /
// tiles: FP64 64^2 1.93 / 1.34, 129^2 3.08 / 1.57, 150 x 600 4.17 / 2.85, but
// 300 x 500 4.30 / 4.37; FP32 129^2 2.94 / 1.66, 300 x 500 4.28 / 2.77, but
// 500^2 4.79 / 6.5; FP16 64^2 1.82 / 2.00 (the cluster kernel), 129^2
// 2.96 / 1.97, 256 x 1024 6.19 / 4.72, 500 x 800 7.51 / 7.28; partially
// saturated obstacles 100 x 250 3.28 / 2.14, but 150 x 600 3.81 / 4.28.
bool tile_plan(int storage, int R, int C, bool partial, int sm_count, TilePlan* plan) {
    *plan = TilePlan{};
    const int form = partial ? 3 : storage == LLB_STORE_F64 ? 0 : storage == LLB_STORE_F32S ? 1 : 2;
    static constexpr long long kMost[4] = {115000, 200000, 400000, 50000}, kLeast[4] = {0, 0, 8000, 0};
    const long long nodes = static_cast<long long>(R) * C;
    if (nodes > kMost[form] || nodes < kLeast[form]) return false;
    const int rpl = form == 1 ? 2 : form == 2 ? 4 : 1;
    // registers per thread of the kernels (columns per warp 1, 2)
    static constexpr int kRegs[4][2] = {{84, 126}, {120, 104}, {126, 128}, {128, 128}};
    double best = 1e30;
    for (int T : {3, 4, 5, 6, 8})
        for (int cpw : {1, 2})
            for (int nw = 8; nw <= 16; nw += 2) {
                const int H = (T + rpl - 1) / rpl * rpl, V = 32 * rpl - 2 * H, TJ = nw * cpw - 2 * T;
                if (TJ < 2) continue;
                const long long tiles = static_cast<long long>((R + V - 1) / V) * ((C + TJ - 1) / TJ);
                const int resident = std::max(1, std::min(64 / nw, 65536 / (kRegs[form][cpw - 1] * 32 * nw)));
                const long long per_sm = (tiles + sm_count - 1) / sm_count;
                const double waves = static_cast<double>((per_sm + resident - 1) / resident);
                const double columns = static_cast<double>(std::min<long long>(per_sm, resident)) * (nw * cpw - T);
                const double step = std::max(0.1 + 0.4 * cpw, 0.05 * columns);
                const double t = (1.2 + waves * (0.3 + T * step)) / T;
                if (t < best) {
                    best = t;
                    *plan = TilePlan{T, H, TJ, cpw};
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
