// Rows of a lattice column held by a lane, and the update of a column of them:
// shared by the kernels that keep populations in registers (llb_stream.cuh,
// llb_tile.cuh).
//
// A lane holds RPL consecutive rows of a column, eight bytes of a population
// plane (or N times that) in every storage form; the rows' neighbours come
// from the neighbouring lanes by shuffles.
#pragma once

#include <type_traits>

#include "llb_kernels.cuh"

namespace llb {

// RPL rows of one population of one lane: N units of eight bytes, as NG groups
// of RG rows that the arithmetic takes at a time (FP64 one row, the shifted
// forms two).
template <class M, int N>
struct Rows;

template <int N>
struct Rows<ModelF64, N> {
    static constexpr int RPL = N, RG = 1, NG = N;
    using V = double;  // a group in the arithmetic type
    using M = ModelF64;
    double v[N];
    static __device__ __forceinline__ Rows load(const void* p) {
        Rows r;
        if constexpr (N == 2) {
            const double2 a = *static_cast<const double2*>(p);
            r.v[0] = a.x;
            r.v[1] = a.y;
        } else {
            r.v[0] = *static_cast<const double*>(p);
        }
        return r;
    }
    __device__ __forceinline__ void store(void* p) const {
        if constexpr (N == 2) *static_cast<double2*>(p) = make_double2(v[0], v[1]);
        else *static_cast<double*>(p) = v[0];
    }
    static __device__ __forceinline__ Rows keep(int k) {
        Rows r;
#pragma unroll
        for (int q = 0; q < N; ++q) r.v[q] = w_init(k);
        return r;
    }
    __device__ __forceinline__ V group(int g) const { return v[g]; }
    __device__ __forceinline__ void set_group(int g, V x) { v[g] = x; }
    // values of the rows above (i - 1) / below (i + 1)
    __device__ __forceinline__ Rows above() const {
        Rows r;
        r.v[0] = __shfl_up_sync(0xffffffffu, v[N - 1], 1);
#pragma unroll
        for (int q = 1; q < N; ++q) r.v[q] = v[q - 1];
        return r;
    }
    __device__ __forceinline__ Rows below() const {
        Rows r;
        r.v[N - 1] = __shfl_down_sync(0xffffffffu, v[0], 1);
#pragma unroll
        for (int q = 0; q + 1 < N; ++q) r.v[q] = v[q + 1];
        return r;
    }
    // rows whose bit k - 1 of their bounce byte is set take own's value
    __device__ __forceinline__ void bounce(unsigned bb, int k, const Rows& own) {
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = ((bb >> (8 * q + k - 1)) & 1u) ? own.v[q] : v[q];
    }
    // rows whose byte in `off` is not zero take the initial value
    __device__ __forceinline__ void reset(unsigned off, int k) {
#pragma unroll
        for (int q = 0; q < N; ++q) v[q] = ((off >> (8 * q)) & 1u) ? w_init(k) : v[q];
    }
    // arithmetic on a group: the density (in the model's form), the divisor of
    // the velocity and its inverse, velocity, collision
    static __device__ __forceinline__ V density(const V* s) { return M::density(s); }
    static __device__ __forceinline__ V divisor(V rr) { return rr; }
    static constexpr bool HAS_MID = false;
    static __device__ __forceinline__ V inverse(V d) { return 1.0 / d; }
    static __device__ __forceinline__ void velocity(const V* s, V inv, V& x, V& y) { M::velocity(s, inv, x, y); }
    template <int COLL>
    static __device__ __forceinline__ void collide(V* s, V rr, V x, V y, const Collision& c) {
        M::collide<COLL>(s, rr, x, y, c);
    }
    static __device__ __forceinline__ bool finite(V rr) { return isfinite(rr); }
    // one row of a group
    static __device__ __forceinline__ double at(V a, int) { return a; }
    static __device__ __forceinline__ void put(V& a, int, double x) { a = x; }
};

// Packed FP32 arithmetic on two rows at a time, common to the shifted forms.
template <class TS>
struct ShiftGroups {
    static constexpr int RG = 2;
    using V = Two::V;
    using M = ModelShift<TS>;
    static __device__ __forceinline__ V density(const V* s) { return M::template density_of<Two>(s); }
    static __device__ __forceinline__ V divisor(V rr) { return Two::add(Two::all(1.0f), rr); }
    static constexpr bool HAS_MID = true;
    static __device__ __forceinline__ bool mid(V d) { return Two::mid(d); }
    static __device__ __forceinline__ V inverse_mid(V d) { return Two::inverse_mid(d); }
    static __device__ __forceinline__ V inverse(V d) { return Two::inverse(d); }
    static __device__ __forceinline__ void velocity(const V* s, V inv, V& x, V& y) {
        M::template velocity_of<Two>(s, inv, x, y);
    }
    template <int COLL>
    static __device__ __forceinline__ void collide(V* s, V rr, V x, V y, const Collision& c) {
        M::template collide_of<COLL, Two>(s, rr, x, y, c);
    }
    static __device__ __forceinline__ bool finite(V rr) {
        const float2 a = Two::unpack(rr);
        return isfinite(a.x) && isfinite(a.y);
    }
    static __device__ __forceinline__ float at(V a, int q) {
        const float2 b = Two::unpack(a);
        return (q & 1) ? b.y : b.x;
    }
    static __device__ __forceinline__ void put(V& a, int q, float x) {
        const float2 b = Two::unpack(a);
        a = Two::pack((q & 1) ? b.x : x, (q & 1) ? x : b.y);
    }
};

template <int N>
struct Rows<ModelShift<float>, N> : ShiftGroups<float> {
    static constexpr int RPL = 2 * N, NG = N;
    V v[N];  // rows 2 n, 2 n + 1 in v[n]
    static __device__ __forceinline__ Rows load(const void* p) {
        Rows r;
        if constexpr (N == 2) {
            const ulonglong2 a = *static_cast<const ulonglong2*>(p);
            r.v[0] = a.x;
            r.v[1] = a.y;
        } else {
            r.v[0] = *static_cast<const unsigned long long*>(p);
        }
        return r;
    }
    __device__ __forceinline__ void store(void* p) const {
        if constexpr (N == 2) *static_cast<ulonglong2*>(p) = make_ulonglong2(v[0], v[1]);
        else *static_cast<unsigned long long*>(p) = v[0];
    }
    static __device__ __forceinline__ Rows keep(int) {
        Rows r;
#pragma unroll
        for (int n = 0; n < N; ++n) r.v[n] = 0ull;
        return r;
    }
    __device__ __forceinline__ V group(int g) const { return v[g]; }
    __device__ __forceinline__ void set_group(int g, V x) { v[g] = x; }
    __device__ __forceinline__ Rows above() const {
        Rows r;
        float last = __shfl_up_sync(0xffffffffu, Two::unpack(v[N - 1]).y, 1);
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const float2 a = Two::unpack(v[n]);
            r.v[n] = Two::pack(last, a.x);
            last = a.y;
        }
        return r;
    }
    __device__ __forceinline__ Rows below() const {
        Rows r;
        float next = __shfl_down_sync(0xffffffffu, Two::unpack(v[0]).x, 1);
#pragma unroll
        for (int n = N - 1; n >= 0; --n) {
            const float2 a = Two::unpack(v[n]);
            r.v[n] = Two::pack(a.y, next);
            next = a.x;
        }
        return r;
    }
    __device__ __forceinline__ void bounce(unsigned bb, int k, const Rows& own) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const float2 a = Two::unpack(v[n]), o = Two::unpack(own.v[n]);
            v[n] = Two::pack(((bb >> (16 * n + k - 1)) & 1u) ? o.x : a.x, ((bb >> (16 * n + k + 7)) & 1u) ? o.y : a.y);
        }
    }
    __device__ __forceinline__ void reset(unsigned off, int) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const float2 a = Two::unpack(v[n]);
            v[n] = Two::pack(((off >> (16 * n)) & 1u) ? 0.0f : a.x, ((off >> (16 * n + 8)) & 1u) ? 0.0f : a.y);
        }
    }
};

template <int N>
struct Rows<ModelShift<__half>, N> : ShiftGroups<__half> {
    static constexpr int RPL = 4 * N, NG = 2 * N;
    uint32_t v[2 * N];  // rows 2 n, 2 n + 1 in v[n]
    static __device__ __forceinline__ Rows load(const void* p) {
        Rows r;
        if constexpr (N == 2) {
            const uint4 u = *static_cast<const uint4*>(p);
            r.v[0] = u.x;
            r.v[1] = u.y;
            r.v[2] = u.z;
            r.v[3] = u.w;
        } else {
            const uint2 u = *static_cast<const uint2*>(p);
            r.v[0] = u.x;
            r.v[1] = u.y;
        }
        return r;
    }
    __device__ __forceinline__ void store(void* p) const {
        if constexpr (N == 2) *static_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
        else *static_cast<uint2*>(p) = make_uint2(v[0], v[1]);
    }
    static __device__ __forceinline__ Rows keep(int) {
        Rows r;
#pragma unroll
        for (int n = 0; n < 2 * N; ++n) r.v[n] = 0u;
        return r;
    }
    __device__ __forceinline__ V group(int g) const {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v[g]));
        return Two::pack(f.x, f.y);
    }
    __device__ __forceinline__ void set_group(int g, V x) {
        const float2 f = Two::unpack(x);
        const __half2 h = __floats2half2_rn(f.x, f.y);
        v[g] = *reinterpret_cast<const uint32_t*>(&h);
    }
    __device__ __forceinline__ Rows above() const {
        Rows r;
        uint32_t last = __shfl_up_sync(0xffffffffu, v[2 * N - 1], 1);
#pragma unroll
        for (int n = 0; n < 2 * N; ++n) {
            r.v[n] = __byte_perm(last, v[n], 0x5432);
            last = v[n];
        }
        return r;
    }
    __device__ __forceinline__ Rows below() const {
        Rows r;
        uint32_t next = __shfl_down_sync(0xffffffffu, v[0], 1);
#pragma unroll
        for (int n = 2 * N - 1; n >= 0; --n) {
            r.v[n] = __byte_perm(v[n], next, 0x5432);
            next = v[n];
        }
        return r;
    }
    template <class B>
    __device__ __forceinline__ void bounce(B bb, int k, const Rows& own) {
#pragma unroll
        for (int h = 0; h < N; ++h) {
            const uint32_t t = ((static_cast<uint32_t>(bb >> (32 * h * (N - 1))) >> (k - 1)) & 0x01010101u) * 0xffu;  // a byte per row
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const uint32_t m = __byte_perm(t, 0u, e == 0 ? 0x1100 : 0x3322);
                v[2 * h + e] = (own.v[2 * h + e] & m) | (v[2 * h + e] & ~m);
            }
        }
    }
    template <class B>
    __device__ __forceinline__ void reset(B off, int) {
#pragma unroll
        for (int h = 0; h < N; ++h) {
            const uint32_t t = static_cast<uint32_t>(off >> (32 * h * (N - 1)));
            v[2 * h] &= ~__byte_perm(t, 0u, 0x1100);
            v[2 * h + 1] &= ~__byte_perm(t, 0u, 0x3322);
        }
    }
};

// One lane's rows of the node masks or bounce bytes, a byte each.
template <int RPL>
struct RowBytes {
    using type = uint32_t;
};
template <>
struct RowBytes<8> {
    using type = unsigned long long;
};
template <int RPL>
__device__ __forceinline__ typename RowBytes<RPL>::type load_row_bytes(const uint8_t* p, unsigned long long pol) {
    typename RowBytes<RPL>::type v;
    if constexpr (RPL == 1) asm("ld.global.nc.L2::cache_hint.u8 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    else if constexpr (RPL == 2) asm("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    else if constexpr (RPL == 4) asm("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    else asm("ld.global.nc.L2::cache_hint.u64 %0, [%1], %2;" : "=l"(v) : "l"(p), "l"(pol));
    return v;
}
// b repeated in every byte of a lane's rows
template <int RPL>
__device__ __forceinline__ constexpr typename RowBytes<RPL>::type each_row(unsigned b) {
    typename RowBytes<RPL>::type v = 0;
    for (int q = 0; q < RPL; ++q) v = (v << 8) | b;
    return v;
}

// 0xff in the byte of every row whose node mask is not active (fluid or open:
// the two class bits 01 or 11, that is bit 0 set).
template <int RPL, class B>
__device__ __forceinline__ B inactive_rows(B m) {
    return (~m & each_row<RPL>(1u)) * static_cast<B>(0xff);
}

// One column of one warp: f = the populations after step t's collision from s,
// the pulled ones (bounce-back done), row q of the lane at (i0 + q, j).
// PLAIN: every row of the warp is a PLAIN fluid node.  SOME: the caller knows
// that at least one row of the lane is active.  mw: the rows' mask bytes.  pol:
// the policy of the open nodes' table reads.  flag: non-finite densities of this
// lane's fluid rows are reported in bad.  out(x, rr, xr, yr): the populations,
// density and velocity of every group, before the collision.
template <class M, int COLL, bool PLAIN, bool SOME, class P, class B, class Out>
__device__ __forceinline__ void update_rows(const Geometry& g, const OpenTable& ot, const Collision& c, const P* s,
                                            P* f, B mw, int i0, int j, long long t, HeldPolicy pol, bool flag,
                                            bool& bad, Out out) {
    using V = typename P::V;
    using R = typename M::R;
    constexpr int NG = P::NG, RG = P::RG, RPL = P::RPL;
    V x[NG][9];
#pragma unroll
    for (int q = 0; q < NG; ++q)
#pragma unroll
        for (int k = 0; k < 9; ++k) x[q][k] = s[k].group(q);
    [[maybe_unused]] V orr[NG], oxr[NG], oyr[NG];  // density and velocity of open rows
    [[maybe_unused]] B open_rows = 0;              // class bits 11
    if constexpr (!PLAIN) {
        open_rows = mw & (mw >> 1) & each_row<RPL>(1u);
        if (open_rows != 0) {
#pragma unroll 1
            for (int q = 0; q < RPL; ++q) {
                const uint8_t m = static_cast<uint8_t>(mw >> (8 * q));
                if (mask_class(m) != CLS_OPEN) continue;
                const int gq = q / RG;
                R y[9];
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    V v = x[0][k];
#pragma unroll
                    for (int n = 1; n < NG; ++n) v = n == gq ? x[n][k] : v;
                    y[k] = P::at(v, q);
                }
                double rho, ux, uy;
                open_node<M>(ot, open_index(g, static_cast<long long>(j) * g.ld + i0 + q, pol), m, t, y, rho, ux, uy,
                             pol);
#pragma unroll
                for (int n = 0; n < NG; ++n)
                    if (n == gq) {
#pragma unroll
                        for (int k = 0; k < 9; ++k) P::put(x[n][k], q, y[k]);
                        P::put(orr[n], q, M::from_f64(rho));
                        P::put(oxr[n], q, static_cast<R>(ux));
                        P::put(oyr[n], q, static_cast<R>(uy));
                    }
            }
        }
    }
    // every group's density and its inverse first (divisions split the code),
    // then the rest, which overlaps
    V rr[NG], iv[NG], xr[NG], yr[NG];
#pragma unroll
    for (int q = 0; q < NG; ++q) {
        rr[q] = P::density(x[q]);
        iv[q] = P::divisor(rr[q]);
    }
    if constexpr (P::HAS_MID) {
        bool mid = true;
#pragma unroll
        for (int q = 0; q < NG; ++q) mid = mid && P::mid(iv[q]);
        if (mid) {
#pragma unroll
            for (int q = 0; q < NG; ++q) iv[q] = P::inverse_mid(iv[q]);
        } else {
#pragma unroll 1
            for (int q = 0; q < NG; ++q)
#pragma unroll
                for (int n = 0; n < NG; ++n)
                    if (n == q) iv[n] = P::inverse(iv[n]);
        }
    } else {
#pragma unroll
        for (int q = 0; q < NG; ++q) iv[q] = P::inverse(iv[q]);
    }
#pragma unroll
    for (int q = 0; q < NG; ++q) P::velocity(x[q], iv[q], xr[q], yr[q]);
    if constexpr (PLAIN) {
#pragma unroll
        for (int q = 0; q < NG; ++q) bad |= flag && !P::finite(rr[q]);
    } else {
#pragma unroll
        for (int q = 0; q < RPL; ++q) {
            const bool fluid = mask_class(static_cast<uint8_t>(mw >> (8 * q))) == CLS_FLUID;
            bad |= flag && fluid && !isfinite(P::at(rr[q / RG], q));
        }
        if (open_rows != 0) {
#pragma unroll
            for (int q = 0; q < RPL; ++q)
                if ((open_rows >> (8 * q)) & 1u) {
                    P::put(rr[q / RG], q, P::at(orr[q / RG], q));
                    P::put(xr[q / RG], q, P::at(oxr[q / RG], q));
                    P::put(yr[q / RG], q, P::at(oyr[q / RG], q));
                }
        }
    }
    out(x, rr, xr, yr);
#pragma unroll
    for (int q = 0; q < NG; ++q) {
        P::template collide<COLL>(x[q], rr[q], xr[q], yr[q], c);
#pragma unroll
        for (int k = 0; k < 9; ++k) f[k].set_group(q, x[q][k]);
    }
    if constexpr (!PLAIN) {
        const B off = inactive_rows<RPL>(mw);
        if (!SOME || (RPL > 1 && off != 0)) {
#pragma unroll
            for (int k = 0; k < 9; ++k) f[k].reset(off, k);
        }
    }
}

}  // namespace llb
