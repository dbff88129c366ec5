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

// Columns of a task.  w: columns each resident warp would walk if the work were
// spread evenly.  Up to 24: one wave of equal tasks (cavity 1000^2 FP64, w = 16:
// 17.3 us a step against 19.2 us in tasks of 12 columns and 21.9 us of 24).
// Above: several waves of smaller tasks, which the block scheduler balances
// (cavity 4096^2 FP64, w = 256, cj = 28: 212 us against 247 us in one wave and
// 230 us in tasks of 12 columns, whose four extra columns weigh more).  Edge
// strips (long path in every column) run chunks half as wide.
template <class CFG>
StreamTasks stream_tasks(int rows, int cols, long long ld, int sm_count) {
    constexpr int EDGE = 2;
    StreamTasks tk{};
    tk.strips = (rows + CFG::V - 1) / CFG::V;
    const double units = std::max(tk.strips - 2, 0) + EDGE * std::min(tk.strips, 2);
    const double w = units * cols / (static_cast<double>(sm_count) * CFG::MB);
    const double cj = w <= 24.0 ? w : std::max(12.0, std::sqrt(3.0 * w));
    tk.cj = std::min(cols, std::max(4, static_cast<int>(std::ceil(cj))));
    // a task's column offsets are 32-bit byte offsets
    tk.cj = static_cast<int>(std::max(1LL, std::min<long long>(tk.cj, (1LL << 31) / (ld * CFG::ES))));
    tk.chunks = (cols + tk.cj - 1) / tk.cj;
    tk.cje = (tk.cj + EDGE - 1) / EDGE;
    tk.chunks_e = (cols + tk.cje - 1) / tk.cje;
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
// 124 us).  The second has the other warp count, the third 16 bytes per lane
// (half the redundant rows, but twice the state: 8 warps per SM).
template <class M, int H, int MB>
cudaError_t step_stream(int cfg, const LaunchCtx& x, const CUtensorMap* pm, void* fout, int sm) {
    switch (cfg - FIRST_STREAM_CONFIG) {
    case 0: return do_step_stream<M, StreamCfg<M, 1, H, 4, MB>>(x, pm, fout, sm);
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
