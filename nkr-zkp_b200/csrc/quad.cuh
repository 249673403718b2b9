// Points held by four lanes.  Lane role r = lane & 3 keeps coordinate r of an XYZZ
// point (0: X, 1: Y, 2: ZZ, 3: ZZZ) and the four lanes compute one product each at a
// time: an addition's 14 products take 4 steps, a doubling's 9 take 3, with the operands
// exchanged by shuffles between the steps.
//
// This is for chains of dependent additions run by few threads (bucket reduction,
// fix-ups, Horner passes, blinding), where a field product is pure latency
// (about 440 ns for a warp alone on its scheduler): one addition by one thread took
// 5 to 8 us there, by four lanes about 2 us.  A lane keeps one coordinate of each
// point, so the G2 forms need no local memory either (one thread holding whole G2
// points spilled up to 2.5 KB).
//
// The formulas are those of curve.cuh (add-2008-s, dbl-2008-s-1) with the
// same treatment of infinity (ZZ = 0), equal and opposite points.  All four lanes of a
// quad take every branch together; other quads of the warp may be elsewhere.
#pragma once

#include "curve.cuh"

namespace nkr {

__device__ __forceinline__ unsigned quad_role() { return threadIdx.x & 3u; }
__device__ __forceinline__ unsigned quad_mask() { return 0xfu << (threadIdx.x & 28u); }

// coordinate of the quad's lane src
template <class P>
__device__ __forceinline__ Fp<P> quad_get(const Fp<P> &a, int src)
{
    Fp<P> r;
#pragma unroll
    for (int j = 0; j < 8; ++j) r.v[j] = __shfl_sync(quad_mask(), a.v[j], src, 4);
    return r;
}
__device__ __forceinline__ FqL quad_get(const FqL &a, int src)
{
    FqL r;
#pragma unroll
    for (int j = 0; j < 8; ++j) r.v[j] = __shfl_sync(quad_mask(), a.v[j], src, 4);
    return r;
}
__device__ __forceinline__ Fq2L quad_get(const Fq2L &a, int src)
{
    Fq2L r;
    r.c0 = quad_get(a.c0, src);
    r.c1 = quad_get(a.c1, src);
    return r;
}

template <class C>
__device__ __forceinline__ C select(bool c, const C &a, const C &b)
{
    return c ? a : b;
}

__device__ __forceinline__ bool quad_flag(bool f, int src) { return __shfl_sync(quad_mask(), int(f), src, 4) != 0; }

// infinity as a quad: X = 0, Y = 1, ZZ = ZZZ = 0
template <class C>
__device__ __forceinline__ C quad_inf()
{
    return quad_role() == 1 ? C::one() : C::zero();
}

template <class C>
__device__ __forceinline__ bool quad_is_inf(const C &v)
{
    return quad_flag(v.is_zero(), 2);
}

// 2 P.  ZZ' = (2Y)^2 ZZ: infinity and points of order two give ZZ' = 0.
template <class C>
__device__ __forceinline__ C quad_dbl(const C &v)
{
    const unsigned role = quad_role();
    const C x = quad_get(v, 0), u = dbl(quad_get(v, 1));
    const C t = select(role == 0, v, u);
    const C s = t * t;                       // lane 0: X^2, others: V = U^2
    const C m = dbl(s) + s;                  // lane 0: M = 3 X^2
    // lane 0: M M, 1: W = U V, 2: ZZ V, 3: S = X V
    const C a = role == 0 ? m : role == 1 ? u : role == 2 ? v : x;
    const C g = a * select(role == 0, m, s);
    const C sx = quad_get(g, 3), w = quad_get(g, 1);
    const C x3 = g - dbl(sx);                // lane 0
    // lane 0: M (S - X'), 1: W Y, 3: W ZZZ
    const C h = select(role == 0, m, w) * select(role == 0, sx - x3, v);
    const C y3 = quad_get(h, 0) - h;         // lane 1
    return role == 0 ? x3 : role == 1 ? y3 : role == 2 ? g : h;
}

// a + b
template <class C>
__device__ __forceinline__ C quad_add(const C &a, const C &b)
{
    if (quad_is_inf(a)) return b;
    if (quad_is_inf(b)) return a;
    const unsigned role = quad_role();
    const int other = int(role ^ 2u);
    // lane 0: U1 = X1 ZZ2, 1: S1 = Y1 ZZZ2, 2: U2 = ZZ1 X2, 3: S2 = ZZZ1 Y2
    const C m = a * quad_get(b, other);
    const C n = quad_get(m, other);
    const bool low = role < 2;
    const C d = select(low, n, m) - select(low, m, n); // P in lanes 0, 2; R in 1, 3
    const bool z = d.is_zero();
    if (quad_flag(z, 0)) return quad_flag(z, 1) ? quad_dbl(a) : quad_inf<C>();
    // lane 0: PP, 1: RR, 2: ZZ1 ZZ2, 3: ZZZ1 ZZZ2
    const C s = select(low, d, a) * select(low, d, b);
    // lane 0: Q = U1 PP, 1 and 3: PPP = P PP, 2: ZZ' = ZZ12 PP
    const C pp = quad_get(s, 0), p = quad_get(d, 0);
    const C g = (role == 0 ? m : role == 2 ? s : p) * pp;
    const C rr = quad_get(s, 1), ppp = quad_get(g, 1), r = quad_get(d, 1);
    const C x3 = rr - ppp - dbl(g);          // lane 0
    // lane 0: R (Q - X'), 1: S1 PPP, 3: ZZZ' = ZZZ12 PPP
    const C h = (role == 0 ? r : role == 1 ? m : s) * select(role == 0, g - x3, g);
    const C y3 = quad_get(h, 0) - h;         // lane 1
    return role == 0 ? x3 : role == 1 ? y3 : role == 2 ? g : h;
}

} // namespace nkr
