// Several steps of a lattice that fits L2 in one launch: overlapped tiles held
// in registers.
//
// One step of such a lattice costs about 3 us whatever its size: a launch, a
// ramp-up, one memory round trip and a drain around well under a microsecond
// of work.  Here a block owns a tile of V rows x TJ columns, loads it with a
// halo of `steps` nodes on every side, advances the whole region `steps` steps,
// and writes the tile back.  Each step the region that is still right shrinks
// by one node on every side.  Blocks never talk to each other, so there is
// nothing to wait for; the halo nodes are computed again by the neighbouring
// tiles, which is what the saved launches pay for.
//
// A warp holds CPW whole columns of the region in registers (32 * RPL rows, RPL
// rows per lane).  Row neighbours come from the neighbouring lanes (shuffles),
// column neighbours inside a warp from its registers; only the three
// populations that leave a warp's first and last column go through shared
// memory (two buffers, one block barrier per step).
//
// The update is the one of the streaming kernel (llb_rows.cuh): the bits are
// those of single steps.  Partially saturated obstacles (PS, FP64): the value a
// fluid node writes into the obstacle's slot comes back to the same node on
// the next step, so between the steps of a launch it stays in shared memory
// beside the node.
//
// What bounds it (B200, cavity 129^2 FP64, 5 steps a launch: 1.57 us a step
// against 3.08 us one step a launch): 1.9 us per launch, and per step the
// instructions of the block that holds the lid (16 warps on the long path,
// each with one open node: 1.2 us; without open nodes 0.8 us).  A version that
// kept both population buffers of the region in shared memory, a thread per
// node, ran 1.72 us a step there and 2.0 us on 181 x 333 FP64.  Four columns per
// warp are slower on all but the largest lattices of the range.
#pragma once

#include "llb_rows.cuh"

namespace llb {

constexpr int TILE_MAX_WARPS = 16;  // per block: 128 registers a thread

// Bytes of shared memory of a block of nw warps.
__host__ __device__ constexpr int tile_smem_bytes(int nw, int cpw, bool ps) {
    return nw * 2 * 6 * 32 * 8 + (ps ? nw * cpw * 8 * 32 * 8 : 0);
}

template <class M, int COLL, int CPW, bool PS>
__global__ void __launch_bounds__(32 * TILE_MAX_WARPS)
    k_step_tile(Geometry g, OpenTable ot, Collision c, const typename M::T* __restrict__ fin,
                typename M::T* __restrict__ fout, MacroOut mo, StepSync ss, int steps, int H, int TJ, int macro) {
    using T = typename M::T;
    using P = Rows<M, 1>;
    using V = typename P::V;
    constexpr int RPL = P::RPL;
    using B = typename RowBytes<RPL>::type;
    constexpr B PLAIN_ALL = each_row<RPL>(CLS_FLUID | MASK_PLAIN), PLAIN_SEL = each_row<RPL>(3u | MASK_PLAIN);
    extern __shared__ __align__(128) unsigned char tile_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int RC = TJ + 2 * steps;  // columns of the region (the last warp may hold more)
    const int j0 = static_cast<int>(blockIdx.y) * TJ - steps + w * CPW;  // this warp's first column
    const int i0 = static_cast<int>(blockIdx.x) * (32 * RPL - 2 * H) - H + lane * RPL;
    const bool row_in = i0 >= 0 && i0 < g.ld;
    const bool own_rows = lane >= H / RPL && lane < 32 - H / RPL && i0 < g.rows;
    // exchange: ex[buffer][warp][0..2] the first column's directions 3, 6, 7
    // (for the left neighbour), [3..5] the last column's 1, 5, 8
    unsigned char* const ex = tile_smem + lane * 8;
    auto slot = [&](int buf, int warp, int n) { return ex + ((buf * nw + warp) * 6 + n) * 256; };
    [[maybe_unused]] double* const vb = reinterpret_cast<double*>(tile_smem + nw * 2 * 6 * 256) + lane;

    B mw[CPW], bw[CPW];
    [[maybe_unused]] unsigned pw[CPW];
    bool pl[CPW];
    const unsigned long long pol = l2_keep_policy();
    const HeldPolicy held{pol};
#pragma unroll
    for (int q = 0; q < CPW; ++q) {
        const int j = j0 + q;
        mw[q] = 0;
        bw[q] = 0;
        if constexpr (PS) pw[q] = 0;
        if (row_in && j >= 0 && j < g.cols) {
            const long long node = static_cast<long long>(j) * g.ld + i0;
            mw[q] = load_row_bytes<RPL>(g.mask + node, pol);
            bw[q] = load_row_bytes<RPL>(g.bb + node, pol);
            if constexpr (PS) pw[q] = g.ps[node];
        }
        pl[q] = __all_sync(0xffffffffu, (mw[q] & PLAIN_SEL) == PLAIN_ALL);
    }
    pdl_wait_then_release();
    const long long t0 = current_step(ss);
    P f[CPW][9];
#pragma unroll
    for (int q = 0; q < CPW; ++q) {
        const int j = j0 + q;
        if (row_in && j >= 0 && j < g.cols) {
            const long long node = static_cast<long long>(j) * g.ld + i0;
#pragma unroll
            for (int k = 0; k < 9; ++k) f[q][k] = P::load(fin + (k * g.plane + node));
            if constexpr (PS) {
#pragma unroll
                for (int k = 1; k < 9; ++k)
                    if ((pw[q] >> (k - 1)) & 1u)
                        vb[((w * CPW + q) * 8 + k - 1) * 32] = fin[k * g.plane + node - (DJ(k) * g.ld + DI(k))];
            }
        } else {
#pragma unroll
            for (int k = 0; k < 9; ++k) f[q][k] = P::keep(k);
        }
        if (!pl[q]) {
            const B off = inactive_rows<RPL>(mw[q]);
#pragma unroll
            for (int k = 0; k < 9; ++k) f[q][k].reset(off, k);
        }
    }

    bool bad = false;
    for (int s = 0; s < steps; ++s) {
        const int buf = s & 1;
        const bool last = s + 1 == steps;
        f[0][3].store(slot(buf, w, 0));
        f[0][6].store(slot(buf, w, 1));
        f[0][7].store(slot(buf, w, 2));
        f[CPW - 1][1].store(slot(buf, w, 3));
        f[CPW - 1][5].store(slot(buf, w, 4));
        f[CPW - 1][8].store(slot(buf, w, 5));
        __syncthreads();
        const int wl = w > 0 ? w - 1 : 0, wr = w + 1 < nw ? w + 1 : w;
        P c1 = P::load(slot(buf, wl, 3)), c5 = P::load(slot(buf, wl, 4)), c8 = P::load(slot(buf, wl, 5));
#pragma unroll
        for (int q = 0; q < CPW; ++q) {
            const int rc = w * CPW + q;  // column of the region
            P s9[9], n1 = f[q][1], n5 = f[q][5], n8 = f[q][8];
            if (rc > s && rc < RC - 1 - s) {  // still right after this step
                s9[0] = f[q][0];
                s9[1] = c1;
                s9[2] = f[q][2].below();
                s9[4] = f[q][4].above();
                s9[5] = c5.below();
                s9[8] = c8.above();
                if (q + 1 < CPW) {
                    s9[3] = f[q + 1 < CPW ? q + 1 : q][3];
                    s9[6] = f[q + 1 < CPW ? q + 1 : q][6].below();
                    s9[7] = f[q + 1 < CPW ? q + 1 : q][7].above();
                } else {
                    s9[3] = P::load(slot(buf, wr, 0));
                    s9[6] = P::load(slot(buf, wr, 1)).below();
                    s9[7] = P::load(slot(buf, wr, 2)).above();
                }
                const int j = j0 + q;
                const bool mine = last && own_rows && rc >= steps && rc < RC - steps && j < g.cols;
                // rho and u of the lane's rows on an output step; 1 and 0 off active nodes
                auto fields = [&](auto value) {
                    if (!(macro && mine)) return;
                    const long long N = static_cast<long long>(g.rows) * g.cols;
#pragma unroll
                    for (int r = 0; r < RPL; ++r)
                        if (i0 + r < g.rows) {
                            const bool act = class_active(mask_class(static_cast<uint8_t>(mw[q] >> (8 * r))));
                            const long long d = static_cast<long long>(j) * g.rows + i0 + r;
                            mo.rho[d] = act ? value(0, r) : 1.0;
                            mo.u[d] = act ? value(1, r) : 0.0;
                            mo.u[d + N] = act ? value(2, r) : 0.0;
                        }
                };
                auto out = [&](const V (*x)[9], const V* rr, const V* xr, const V* yr) {
                    fields([&](int n, int r) {
                        return n == 0   ? M::rho_f64(P::at(rr[r / P::RG], r))
                               : n == 1 ? static_cast<double>(P::at(xr[r / P::RG], r))
                                        : static_cast<double>(P::at(yr[r / P::RG], r));
                    });
                };
                if (pl[q]) {
                    update_rows<M, COLL, true, true>(g, ot, c, s9, f[q], mw[q], i0, j, t0 + s, held, mine, bad, out);
                } else if (inactive_rows<RPL>(mw[q]) == each_row<RPL>(0xffu)) {
                    fields([](int, int) { return 0.0; });  // no active row: f keeps the initial values
                } else {
                    s9[1].bounce(bw[q], 1, f[q][3]);
                    s9[2].bounce(bw[q], 2, f[q][4]);
                    s9[3].bounce(bw[q], 3, f[q][1]);
                    s9[4].bounce(bw[q], 4, f[q][2]);
                    s9[5].bounce(bw[q], 5, f[q][7]);
                    s9[6].bounce(bw[q], 6, f[q][8]);
                    s9[7].bounce(bw[q], 7, f[q][5]);
                    s9[8].bounce(bw[q], 8, f[q][6]);
                    if constexpr (PS) {
                        double* const v = vb + rc * 8 * 32;
#pragma unroll
                        for (int k = 1; k < 9; ++k)
                            if ((pw[q] >> (k - 1)) & 1u) s9[k].v[0] = v[(k - 1) * 32];
                        double sp[9], prr = 0.0, pxr = 0.0, pyr = 0.0;
                        update_rows<M, COLL, false, true>(g, ot, c, s9, f[q], mw[q], i0, j, t0 + s, held, mine, bad,
                                                    [&](const V (*x)[9], const V* rr, const V* xr, const V* yr) {
                                                        out(x, rr, xr, yr);
#pragma unroll
                                                        for (int k = 0; k < 9; ++k) sp[k] = x[0][k];
                                                        prr = rr[0];
                                                        pxr = xr[0];
                                                        pyr = yr[0];
                                                    });
                        if (pw[q]) {
                            const long long node = static_cast<long long>(j) * g.ld + i0;
                            double fp[9];
#pragma unroll
                            for (int k = 0; k < 9; ++k) fp[k] = f[q][k].v[0];
                            if (!last)
                                ps_push_values(g, node, pw[q], sp, fp, prr, pxr, pyr, c.ps_t,
                                               [&](int k, double x) { v[(k - 1) * 32] = x; });
                            else if (mine)
                                ps_push(g, fout, node, pw[q], sp, fp, prr, pxr, pyr, c.ps_t);
                        }
                    } else {
                        update_rows<M, COLL, false, true>(g, ot, c, s9, f[q], mw[q], i0, j, t0 + s, held, mine, bad, out);
                    }
                }
                if (mine) {
                    const long long node = static_cast<long long>(j) * g.ld + i0;
                    // an obstacle's slots belong to its neighbours
                    if (!PS || class_active(mask_class(static_cast<uint8_t>(mw[q])))) {
#pragma unroll
                        for (int k = 0; k < 9; ++k) f[q][k].store(fout + (k * g.plane + node));
                    }
                }
            }
            c1 = n1;
            c5 = n5;
            c8 = n8;
        }
    }
    flag_numerics(ss, bad);
}

}  // namespace llb
