// Launches of the register-streaming two-step kernel (llb_stream.cuh) for every
// storage form.  Compiled with --fmad=false, like the other step kernels, so
// its arithmetic rounds as theirs.
#include "llb_stream.cuh"

#include <algorithm>
#include <cmath>

#include "../../include/llalbm_cuda.h"
#include "llb_launch.h"
#include "llb_pdl.cuh"

namespace llb {

namespace {

// Columns of a task, four of which it computes or reads besides its own.  w:
// columns each resident warp would walk if the work were spread evenly.
// Up to w = 40: the narrowest tasks that are one wave, none left over for a
// second one.  Against tasks of 12 columns in several waves (us a step): channel
// 1001 x 3005 FP32, w = 25, 26.4 -> 23.6; cavity 2048^2 FP16, w = 24, 32.1 -> 29.5;
// porous 1300^2 FP64 on configuration 3, w = 27, 31.8 -> 28.8; channel 1500 x 3000
// FP32, w = 37, 37.1 -> 34.6.  Above, the slowest task of one wave takes too long
// (cavity 2400^2 FP32, w = 46, 48.3 in one wave): several waves, which the block
// scheduler balances, of sqrt(9 w) columns up to 24 (porous 3600^2 FP32, w = 102,
// 98.7 against 101.9 in tasks of 17 columns; cavity 2900^2 FP32, w = 66, 58.5
// against 59.8 in tasks of 14), and of sqrt(3 w) when that is more (cavity 4096^2
// FP64, w = 258, 28 columns: 212 against 217 in tasks of 48 and 227 in tasks of 24).
// Edge strips (long path in every column) run chunks half as wide.
template <class CFG>
StreamTasks stream_tasks(int rows, int cols, long long ld, int sm_count) {
    constexpr int EDGE = 2;
    StreamTasks tk{};
    tk.strips = (rows + CFG::V - 1) / CFG::V;
    const int edges = std::min(tk.strips, 2), inner = tk.strips - edges;
    const long long room = static_cast<long long>(sm_count) * CFG::MB;
    auto edge_width = [](int c) { return (c + EDGE - 1) / EDGE; };
    auto chunks = [&](int c) { return (cols + c - 1) / c; };
    const double w = static_cast<double>(inner + EDGE * edges) * cols / static_cast<double>(room);
    int cj = std::max(4, static_cast<int>(std::ceil(
                             w <= 40.0 ? w : std::max(std::min(std::sqrt(9.0 * w), 24.0), std::sqrt(3.0 * w)))));
    if (w <= 40.0)
        while (cj < cols && static_cast<long long>(inner) * chunks(cj) + edges * chunks(edge_width(cj)) > room) ++cj;
    tk.cj = std::min(cols, cj);
    // a task's column offsets are 32-bit byte offsets
    tk.cj = static_cast<int>(std::max(1LL, std::min<long long>(tk.cj, (1LL << 31) / (ld * CFG::ES))));
    tk.chunks = chunks(tk.cj);
    tk.cje = edge_width(tk.cj);
    tk.chunks_e = chunks(tk.cje);
    return tk;
}

template <class M, class CFG>
cudaError_t do_step_stream(const LaunchCtx& x, const CUtensorMap* pmap, void* fout, int sm_count) {
    using T = typename M::T;
    const StreamTasks tk = stream_tasks<CFG>(x.g.rows, x.g.cols, x.g.ld, sm_count);
    const int tasks = std::min(tk.strips, 2) * tk.chunks_e + std::max(tk.strips - 2, 0) * tk.chunks;
    auto kern = x.c.model == 0 ? k_step_stream<M, 0, CFG> : k_step_stream<M, 1, CFG>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CFG::SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    return launch_pdl_smem(kern, dim3(tasks), dim3(32), CFG::SMEM_BYTES, x.stream, *pmap, x.g, x.ot, x.c,
                           static_cast<T*>(fout), x.ss, tk);
}

using ModelF32S = ModelShift<float>;
using ModelF16S = ModelShift<__half>;

// Configurations (eight-byte units per lane, halo rows, stages, warps per SM).
// The first is the default: 16 warps of 128 registers per SM, 12 of 168 in FP16,
// whose conversions spill at 128 (cavity 4096^2 FP16: 99 us a step against
// 124 us), and 3 stages (a fourth or fifth takes L1 from the mask bytes: channel
// 1001 x 3005 FP32 23.4 us a step with 3, 23.8 with 4; FP64 the same).  The second
// has the other warp count, the third 16 bytes per lane (half the redundant
// rows, but twice the state: 8 warps per SM).
template <class M, int H, int MB>
cudaError_t step_stream(int cfg, const LaunchCtx& x, const CUtensorMap* pm, void* fout, int sm) {
    switch (cfg - FIRST_STREAM_CONFIG) {
    case 0: return do_step_stream<M, StreamCfg<M, 1, H, 3, MB>>(x, pm, fout, sm);
    case 1: return do_step_stream<M, StreamCfg<M, 1, H, 4, 28 - MB>>(x, pm, fout, sm);
    case 2: return do_step_stream<M, StreamCfg<M, 2, H, 4, 8>>(x, pm, fout, sm);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace

int stream_box_rows(int storage, int cfg) {
    const int lane_bytes = cfg - FIRST_STREAM_CONFIG == 2 ? 16 : 8;
    return 32 * lane_bytes / (storage == LLB_STORE_F64 ? 8 : storage == LLB_STORE_F32S ? 4 : 2);
}

cudaError_t launch_step_stream(int storage, int cfg, const LaunchCtx& x, const CUtensorMap* pmap, void* fout,
                               int sm_count) {
    switch (storage) {
    case LLB_STORE_F64: return step_stream<ModelF64, 2, 16>(cfg, x, pmap, fout, sm_count);
    case LLB_STORE_F32S: return step_stream<ModelF32S, 4, 16>(cfg, x, pmap, fout, sm_count);
    default: return step_stream<ModelF16S, 8, 12>(cfg, x, pmap, fout, sm_count);
    }
}

}  // namespace llb
