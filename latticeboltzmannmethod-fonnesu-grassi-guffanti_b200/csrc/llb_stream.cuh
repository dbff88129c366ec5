// Two steps per pass over HBM, streamed through registers.
//
// A plain step reads and writes the nine populations of every node, so at the
// copy bandwidth its rate is fixed by the bytes per node.  Here a warp owns a
// strip of rows and walks along the columns with NT = 2 time levels in flight:
// it takes column j of f*_{t-1}, computes column j - 1 of f*_t from it and the
// two columns before, column j - 2 of f*_{t+1} from that, and stores it.
// Between two columns a level keeps nine values per row, all in registers: the
// six populations that are already in place for the next level (directions 0,
// 2, 4 from its newest column, 1, 5, 8 from the one before) and the newest
// column's own directions 1, 5, 8.
//
// A block is one warp, so warps share nothing and never wait for each other.
// Columns arrive by TMA: one box of 32 * RPL rows x 1 column x 9 planes per
// column, S stages ahead, in the block's own shared memory.  Each level loses
// one row at either end of the strip: of 32 * RPL rows loaded the inner
// V = 32 * RPL - 2 H are stored (H >= NT; V rows are whole 32-byte sectors and the
// box starts on a 16-byte boundary), and a chunk of columns [c0, c1) starts NT
// columns early and ends NT columns late.  Outside the lattice the boxes read
// zeros and the mask is 0: dead nodes, which get their initial values.
//
// Columns whose nodes (in this strip) are all PLAIN fluid nodes take the short
// path, a warp vote.  The others replace a population whose source is a wall
// or wet obstacle by the node's own opposite one (bounce bits) and give
// inactive nodes the initial values.  A level's populations are rounded to the
// storage type, and the arithmetic per node is the storage model's, so the
// bits are those of two single steps.
//
// What bounds it (B200): FP64 HBM -- cavity 4096^2 212 us a step (two passes of
// nine planes every two steps are 187 us at the copy bandwidth) against 335 us
// for the tile-in-shared-memory kernel this one replaced; FP32 117 us against
// 193 us, FP16 99 us against 141 us, there fixed-latency waits at three and two
// warps per scheduler (2048^2: issue slots 64 and 55 % busy, 1.4 cycles of wait
// an instruction, DRAM 50 and 26 %; porous FP64 65 %, 1.7 and 55 %).  The packed FP32
// arithmetic (Two, llb_model.cuh) halves the instructions of the shifted forms'
// collision; without it FP32 ran 136 us.  Measured and dropped: four levels (the
// state of four levels leaves 8 warps per SM, and FP64 needs 4 halo rows: 320 us,
// FP32 146 us); the column loop unrolled twice (10-30 % slower everywhere: the
// loop no longer fits the instruction cache); plain loads instead of TMA.
//
// The wait for a stage is bounded: on timeout the warp sets FLAG_TIMEOUT, waits
// (bounded) for its copies in flight and returns.
#pragma once

#include "llb_launch.h"
#include "llb_rows.cuh"
#include "llb_tma.cuh"

namespace llb {

// Compile-time shape: N eight-byte units of a plane per lane, H halo rows at
// either end of a strip, S stages, MB resident blocks (warps) per SM.
template <class M, int N_, int H_, int S_, int MB_>
struct StreamCfg {
    static constexpr int N = N_, NT = STREAM_STEPS, H = H_, S = S_, MB = MB_;
    using P = Rows<M, N>;
    static constexpr int RPL = P::RPL;
    static constexpr int ROWS = 32 * RPL;
    static constexpr int V = ROWS - 2 * H;  // rows stored per strip
    static constexpr int LANE_BYTES = 8 * N;
    static constexpr int STAGE_BYTES = 9 * 32 * LANE_BYTES;
    static constexpr int SMEM_BYTES = S * STAGE_BYTES + S * 8;
    static constexpr int ES = LANE_BYTES / RPL;  // bytes of an element
    static_assert(H >= NT && (H * ES) % 16 == 0 && (V * ES) % 32 == 0, "strip shape");
    static_assert(MB * (SMEM_BYTES + 1024) <= 233472, "shared memory per SM");
};

// Tasks of a launch: chunks of cj columns of every strip; the first and the
// last strip (walls and often a whole row of open nodes, so every column takes
// the long path) in chunks of cje columns, first in the launch order.
struct StreamTasks {
    int strips, cj, chunks, cje, chunks_e;
};

template <class M, int COLL, class CFG>
__global__ void __launch_bounds__(32, CFG::MB)
    k_step_stream(const __grid_constant__ CUtensorMap pmap, Geometry g, OpenTable ot, Collision c,
                  typename M::T* __restrict__ fout, StepSync ss, StreamTasks tk) {
    using R = typename M::R;
    using P = typename CFG::P;
    using V = typename P::V;
    constexpr int NT = CFG::NT, H = CFG::H, RPL = CFG::RPL, S = CFG::S, ES = CFG::ES;
    using B = typename RowBytes<RPL>::type;
    constexpr B PLAIN_ALL = each_row<RPL>(CLS_FLUID | MASK_PLAIN), PLAIN_SEL = each_row<RPL>(3u | MASK_PLAIN);
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* const full = reinterpret_cast<uint64_t*>(smem + S * CFG::STAGE_BYTES);
    const int lane = threadIdx.x;

    // this block's strip and columns
    int strip, c0, c1;
    {
        const int edges = min(tk.strips, 2) * tk.chunks_e;
        const int b = static_cast<int>(blockIdx.x);
        if (b < edges) {
            strip = b < tk.chunks_e ? 0 : tk.strips - 1;
            c0 = (b < tk.chunks_e ? b : b - tk.chunks_e) * tk.cje;
            c1 = min(c0 + tk.cje, g.cols);
        } else {
            const int inner = tk.strips - 2, r = b - edges;
            strip = 1 + r % inner;
            c0 = (r / inner) * tk.cj;
            c1 = min(c0 + tk.cj, g.cols);
        }
    }
    const int x0 = strip * CFG::V - H;          // first row of the box
    const int i0 = x0 + lane * RPL;        // first row of this lane
    const int nit = (c1 - c0) + 2 * NT;
    if (lane == 0) {
        for (int s = 0; s < S; ++s) mbar_init(&full[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const bool row_in = i0 >= 0 && i0 < g.ld;
    const bool own_rows = lane >= H / RPL && lane < 32 - H / RPL && i0 < g.rows;
    const unsigned long long pol = l2_keep_policy();
    const HeldPolicy held{pol};
    B nm = 0, nb = 0;  // masks and bounce bytes of the next column
    auto fetch_bytes = [&](int j) {
        nm = 0;
        nb = 0;
        if (row_in && j >= 0 && j < g.cols) {
            const long long node = static_cast<long long>(j) * g.ld + i0;
            nm = load_row_bytes<RPL>(g.mask + node, pol);
            nb = load_row_bytes<RPL>(g.bb + node, pol);
        }
    };
    auto fetch = [&](int s, int j) {  // one lane
        mbar_expect_tx(&full[s], CFG::STAGE_BYTES);
        tma_load_3d(smem + s * CFG::STAGE_BYTES, &pmap, x0, j, 0, &full[s]);
    };
    fetch_bytes(c0 - NT);
    pdl_wait_then_release();
    const long long t0 = current_step(ss);
    if (lane == 0)
        for (int s = 0; s < S && s < nit; ++s) fetch(s, c0 - NT + s);

    // per level: the populations in place for the next level's newest-but-one
    // column (directions 0 1 2 4 5 8) and the newest column's own 1, 5, 8
    P in0[NT], in1[NT], in2[NT], in4[NT], in5[NT], in8[NT], o1[NT], o5[NT], o8[NT];
    B mw[NT + 1], bw[NT + 1];  // masks and bounce bytes of columns j, j - 1, ...
    bool pl[NT + 1];           // warp-uniform: the column's nodes here are all PLAIN fluid nodes
#pragma unroll
    for (int l = 0; l < NT; ++l) {
        in0[l] = P::keep(0); in1[l] = P::keep(1); in2[l] = P::keep(2); in4[l] = P::keep(4);
        in5[l] = P::keep(5); in8[l] = P::keep(8); o1[l] = P::keep(1); o5[l] = P::keep(5); o8[l] = P::keep(8);
    }
#pragma unroll
    for (int l = 0; l <= NT; ++l) { mw[l] = 0; bw[l] = 0; pl[l] = false; }

    bool bad = false;
    int s_at = 0;
    unsigned phase = 0;
    unsigned char* const out0 = reinterpret_cast<unsigned char*>(fout + static_cast<long long>(c0) * g.ld + x0);
    unsigned out_off = static_cast<unsigned>(lane) * static_cast<unsigned>(CFG::LANE_BYTES);  // of this lane's rows in the column being stored
    const unsigned out_step = static_cast<unsigned>(g.ld) * static_cast<unsigned>(ES);
    for (int it = 0; it < nit; ++it) {
        const int j = c0 - NT + it;
        if (!__all_sync(0xffffffffu, mbar_wait(&full[s_at], phase, ss.wait_limit))) {
            if (lane == 0) {
                atomicOr(ss.flags, FLAG_TIMEOUT);
                // do not leave with copies in flight: the stages still outstanding
                for (int q = 0; q < S && it + q < nit; ++q) {
                    const int sq = (s_at + q) % S;
                    if (!mbar_wait(&full[sq], phase ^ (s_at + q >= S ? 1u : 0u))) atomicOr(ss.flags, FLAG_TIMEOUT);
                }
            }
            return;
        }
        P f[9];
        const unsigned char* const st = smem + s_at * CFG::STAGE_BYTES + lane * CFG::LANE_BYTES;
#pragma unroll
        for (int k = 0; k < 9; ++k) f[k] = P::load(st + k * 32 * CFG::LANE_BYTES);
#pragma unroll
        for (int l = NT; l > 0; --l) { mw[l] = mw[l - 1]; bw[l] = bw[l - 1]; pl[l] = pl[l - 1]; }
        mw[0] = nm;
        bw[0] = nb;
        pl[0] = __all_sync(0xffffffffu, (nm & PLAIN_SEL) == PLAIN_ALL);
        fetch_bytes(j + 1);
        if constexpr (sizeof(R) == 8) {
            if (!pl[0]) {  // rows outside the lattice arrive as zeros, not as the initial values
#pragma unroll
                for (int k = 0; k < 9; ++k) f[k].reset(inactive_rows<RPL>(mw[0]), k);
            }
        }
#pragma unroll
        for (int l = 0; l < NT; ++l) {
            // f: column j - l of level l
            if (it < 2 * l) break;  // not reached yet
            P s[9];
            const bool ready = it >= 2 * l + 2;
            // S of column j - l - 1, complete with this column's directions 3, 6, 7
            s[0] = in0[l]; s[1] = in1[l]; s[2] = in2[l]; s[4] = in4[l]; s[5] = in5[l]; s[8] = in8[l];
            s[3] = f[3];
            s[6] = f[6].below();
            s[7] = f[7].above();
            if (!pl[l + 1]) {
                s[3].bounce(bw[l + 1], 3, o1[l]);
                s[6].bounce(bw[l + 1], 6, o8[l]);
                s[7].bounce(bw[l + 1], 7, o5[l]);
            }
            // this column's populations for the next one
            in0[l] = f[0];
            in1[l] = o1[l];
            in2[l] = f[2].below();
            in4[l] = f[4].above();
            in5[l] = o5[l].below();
            in8[l] = o8[l].above();
            if (!pl[l]) {
                in1[l].bounce(bw[l], 1, f[3]);
                in2[l].bounce(bw[l], 2, f[4]);
                in4[l].bounce(bw[l], 4, f[2]);
                in5[l].bounce(bw[l], 5, f[7]);
                in8[l].bounce(bw[l], 8, f[6]);
            }
            o1[l] = f[1];
            o5[l] = f[5];
            o8[l] = f[8];
            if (!ready) break;
            // column j - l - 1 of level l + 1, into f: once for all-PLAIN
            // columns, once for the others
            const int cc = j - l - 1;
            const auto none = [](const V (*)[9], const V*, const V*, const V*) {};
            // (a non-finite density stays one, so the last level's check finds it)
            const bool flag = l + 1 == NT && own_rows;
            if (pl[l + 1]) update_rows<M, COLL, true, false>(g, ot, c, s, f, mw[l + 1], i0, cc, t0 + l, held, flag, bad, none);
            else update_rows<M, COLL, false, false>(g, ot, c, s, f, mw[l + 1], i0, cc, t0 + l, held, flag, bad, none);
            if (l + 1 == NT) {
                if (own_rows) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) f[k].store(out0 + k * g.plane * ES + out_off);
                }
                out_off += out_step;
            }
        }
        // The stage is refilled only here, where every lane has used what it
        // read from it: a load still on its way to registers would race with
        // the copy, which shared-memory loads are not ordered against.
        __syncwarp();
        if (lane == 0 && it + S < nit) fetch(s_at, j + S);
        if (++s_at == S) { s_at = 0; phase ^= 1u; }
    }
    flag_numerics(ss, bad);
}

}  // namespace llb
