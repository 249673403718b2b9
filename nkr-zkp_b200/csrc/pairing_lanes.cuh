// The pairing of pairing.cuh with six lanes per value: lane m of a group holds the
// coefficient a_m in Fq2 of f = sum_m a_m w^m (w^6 = xi), five groups to a warp.
//
// One thread per pairing is latency bound for any batch below some ten thousand pairings
// (a warp per scheduler at 32 K), and its Fq12 values live in local memory (12.8 KB of
// call frames a thread).  With a coefficient per lane a product is one dot product per
// lane, c_k = sum_i a_i b_(k-i) (times xi where the index wraps), whose terms are summed
// as 512-bit integers before a single pair of Montgomery reductions: 6 x 192 + 128 wide
// multiply-adds per lane, against 18 Fq2 products of 384 by one thread.  All arithmetic goes
// through one out-of-line routine (lane_dot), so the hot code is about 10 KB.  Operands
// are exchanged through shared memory; only the lane's own coefficient stays in
// registers.  4,096 verifications (four public inputs, from host memory) took 29.7 ms with
// one thread per proof and take 5.1 ms with six lanes (B200).
//
// Squarings in the final exponentiation's cyclotomic part use Granger and Scott's
// formulas ("Faster squaring in the cyclotomic subgroup of sixth degree extensions", PKC
// 2010) over Fq4 = Fq2[w^3]: two terms instead of four.  Field elements are canonical
// throughout.
#pragma once

#include "pairing.cuh"

namespace nkr {

constexpr int kPairLanes = 6;   // lanes per group
constexpr int kPairGroups = 5;  // groups per warp (lanes 30 and 31 shadow the last one)
// A slot holds one Fq2 in four 16-byte chunks, 5 chunks apart; groups are 246 chunks
// apart (6 mod 8): the eight lanes of a 128-byte access that read consecutive slots of one
// group and of the next touch different banks.
constexpr int kSlotChunks = 5;
constexpr int kGroupChunks = 246;
constexpr int kPairSmemChunks = kPairGroups * kGroupChunks;

// slots of a group
enum PairSlot {
    kSlA = 0,       // 0-5: first operand's coefficients
    kSlXA = 6,      // 6-11: xi times them
    kSlB = 12,      // 12-17: second operand (squarings: 2 A)
    kSlXB = 18,     // 18-23: xi times it (squarings: 2 xi A)
    kSlT = 12,      // 12-23 hold temporaries of the point steps
    kSlLine = 24,   // 5 slots per pair: c0, a, b, xi a, xi b
    kSlX = 39,      // T in homogeneous coordinates
    kSlY = 40,
    kSlZ = 41,
    kSlQx = 42,     // the point added to T
    kSlQy = 43,
    kSlNegPx = 44,  // -xP and yP of pair 0
    kSlPy = 45,
    kSlNegPx1 = 46, // -xP of pairs 1 and 2
    kSlNegPx2 = 47,
    kSlScale1 = 13, // pair 1's line scale (only during the first level of a point step)
    kSlZero = 48,
};

// sums of products as 512-bit integers: even and odd accumulators (mul_wide in
// field.cuh) with the chains' carries counted apart, c[j] at word offset 8 + j
struct WideSum {
    uint32_t e[16], o[14], c[9];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int j = 0; j < 16; ++j) e[j] = 0;
#pragma unroll
        for (int j = 0; j < 14; ++j) o[j] = 0;
#pragma unroll
        for (int j = 0; j < 9; ++j) c[j] = 0;
    }
    __device__ __forceinline__ void add_product(const uint32_t *x, const uint32_t *y)
    {
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            eo_mad(e + i, c[i], x[0], x[2], x[4], x[6], y[i]);
            eo_mad(o + i, c[i + 1], x[1], x[3], x[5], x[7], y[i]);
            eo_mad(o + i, c[i + 1], x[0], x[2], x[4], x[6], y[i + 1]);
            eo_mad(e + i + 2, c[i + 2], x[1], x[3], x[5], x[7], y[i + 1]);
        }
    }
    __device__ __forceinline__ void total(uint32_t *t) const
    {
        uint32_t hi[8], oh[8], carry = 0;
#pragma unroll
        for (int j = 0; j < 6; ++j) oh[j] = o[8 + j];
        oh[6] = oh[7] = 0;
        uint32_t eh[8];
#pragma unroll
        for (int j = 0; j < 7; ++j) eh[j] = e[9 + j];
        eh[7] = 0;
        t[0] = e[0];
        add_words_carry(t + 1, e + 1, o, carry); // words 1..8
        add_words_carry(hi, eh, oh, carry);      // words 9..15
#pragma unroll
        for (int j = 0; j < 7; ++j) t[9 + j] = hi[j];
        add_words(t + 8, t + 8, c);
    }
};

// 6 p^2, 16 little-endian words
__device__ __forceinline__ uint32_t six_p2_word(int k)
{
    constexpr uint32_t w[16] = {0xec307a26u, 0x63fa13ccu, 0x3b808607u, 0xe40c2b0eu, 0x9188c12bu, 0xbde093aau,
                                0xdc6d90b1u, 0x1a73b780u, 0x3ca8354eu, 0xe993de29u, 0x854c0424u, 0x20451fe6u,
                                0x13b4ecacu, 0x199e9ce8u, 0xc56c7daau, 0x36e29c52u};
    return w[k];
}

__device__ __forceinline__ void load_half(const uint4 *p, uint32_t *w)
{
    const uint4 a = p[0], b = p[1];
    w[0] = a.x;
    w[1] = a.y;
    w[2] = a.z;
    w[3] = a.w;
    w[4] = b.x;
    w[5] = b.y;
    w[6] = b.z;
    w[7] = b.w;
}

// T 2^-256 mod p for T <= 12 p^2 (below 2.3 p 2^256): the reduction of the low half adds at
// most p, so the value is below 3.3 p before the two conditional subtractions
__device__ __forceinline__ Fq redc_sum(const uint32_t *t)
{
    uint32_t lo[8];
    Fq r;
    redc_low<FqParams>(t, lo);
    add_words(r.v, lo, t + 8);
    reduce_once<TwoP<FqParams>>(r.v);
    reduce_once<FqParams>(r.v);
    return r;
}

// sum over n terms of slot(a_t) slot(b_t); byte t of ta and of tb names the slots.  The
// operands' coordinates are below 2p and the products sum to at most 6 p^2 per coordinate
// pair (canonical operands: n <= 6; a doubled operand counts twice), so the Karatsuba sum
// of (x0 + x1)(y0 + y1) stays below 24 p^2 < 2^512.
__device__ __noinline__ Fq2 lane_dot(const uint4 *s, int n, uint64_t ta, uint64_t tb)
{
    uint32_t t0[16], t1[16], x[8], y[8];
    WideSum acc;
    acc.clear();
#pragma unroll 1
    for (int t = 0; t < n; ++t) { // sum x1 y1
        load_half(s + int((ta >> (8 * t)) & 255u) * kSlotChunks + 2, x);
        load_half(s + int((tb >> (8 * t)) & 255u) * kSlotChunks + 2, y);
        acc.add_product(x, y);
    }
    acc.total(t1);
    acc.clear();
#pragma unroll 1
    for (int t = 0; t < n; ++t) { // sum x0 y0
        load_half(s + int((ta >> (8 * t)) & 255u) * kSlotChunks, x);
        load_half(s + int((tb >> (8 * t)) & 255u) * kSlotChunks, y);
        acc.add_product(x, y);
    }
    acc.total(t0);
    Fq2 r;
    {
        uint32_t d[16], w[16], c = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = six_p2_word(j);
        add_words_carry(d, t0, w, c);
        add_words_carry(d + 8, t0 + 8, w + 8, c);
        sub_words16(d, d, t1);
        r.c0 = redc_sum(d);
        c = 0;
        add_words_carry(t1, t0, t1, c);
        add_words_carry(t1 + 8, t0 + 8, t1 + 8, c);
    }
    acc.clear();
#pragma unroll 1
    for (int t = 0; t < n; ++t) { // sum (x0 + x1)(y0 + y1)
        uint32_t u[8];
        const uint4 *p = s + int((ta >> (8 * t)) & 255u) * kSlotChunks;
        load_half(p, x);
        load_half(p + 2, u);
        add_words(x, x, u);
        p = s + int((tb >> (8 * t)) & 255u) * kSlotChunks;
        load_half(p, y);
        load_half(p + 2, u);
        add_words(y, y, u);
        acc.add_product(x, y);
    }
    acc.total(t0);
    sub_words16(t0, t0, t1);
    r.c1 = redc_sum(t0);
    return r;
}

// a byte per lane of the group
__device__ __forceinline__ constexpr uint64_t lane_bytes(int b0, int b1, int b2, int b3, int b4, int b5)
{
    return uint64_t(b0) | uint64_t(b1) << 8 | uint64_t(b2) << 16 | uint64_t(b3) << 24 | uint64_t(b4) << 32 |
           uint64_t(b5) << 40;
}
// up to six terms of one lane
__device__ __forceinline__ constexpr uint64_t terms(int t0, int t1 = 0, int t2 = 0, int t3 = 0)
{
    return lane_bytes(t0, t1, t2, t3, 0, 0);
}

// Digit b of z in signed odd digits (width-4 non-adjacent form, 4 bits a digit).  The table
// is local: device code cannot index a host constant of namespace scope at run time.
__host__ __device__ constexpr int z_digit(int b)
{
    const uint64_t w[4] = {0x50000f0001ull, 0x100005000070009ull, 0x300005000b000d00ull, 0x10000050000d000ull};
    return (int(w[b >> 4] >> (4 * (b & 15)) & 15u) ^ 8) - 8;
}
constexpr uint64_t z_of_digits()
{
    uint64_t z = 0;
    for (int b = 0; b < 63; ++b) z += uint64_t(int64_t(z_digit(b))) << b;
    return z;
}
static_assert(z_of_digits() == kZ && z_digit(62) == 1, "digits of z");

struct PairGroup {
    uint4 *s;    // the group's slots
    int m;       // this lane's coefficient
    bool live;   // lanes 30 and 31 store nothing
    uint64_t sqr_a, sqr_b, cyc_a, cyc_b;

    __device__ PairGroup(uint4 *smem, int lane)
    {
        const int l = lane < kPairLanes * kPairGroups ? lane : lane - kPairLanes + 4; // 30, 31 -> 28, 29
        live = lane < kPairLanes * kPairGroups;
        s = smem + (l / kPairLanes) * kGroupChunks;
        m = l % kPairLanes;
        constexpr int A = kSlA, X = kSlXA, D = kSlB, E = kSlXB, Z = kSlZero;
        // c_m of a square: cross terms with a doubled factor, then squares
        switch (m) {
        case 0:
            sqr_a = terms(A + 1, A + 2, A + 3, A);
            sqr_b = terms(E + 5, E + 4, X + 3, A);
            cyc_a = terms(A, A + 3);
            cyc_b = terms(A, X + 3);
            break;
        case 1:
            sqr_a = terms(A, A + 2, A + 3, Z);
            sqr_b = terms(D + 1, E + 5, E + 4, Z);
            cyc_a = terms(A + 2, Z);
            cyc_b = terms(E + 5, Z);
            break;
        case 2:
            sqr_a = terms(A, A + 3, A + 1, A + 4);
            sqr_b = terms(D + 2, E + 5, A + 1, X + 4);
            cyc_a = terms(A + 1, A + 4);
            cyc_b = terms(A + 1, X + 4);
            break;
        case 3:
            sqr_a = terms(A, A + 1, A + 4, Z);
            sqr_b = terms(D + 3, D + 2, E + 5, Z);
            cyc_a = terms(A, Z);
            cyc_b = terms(D + 3, Z);
            break;
        case 4:
            sqr_a = terms(A, A + 1, A + 2, A + 5);
            sqr_b = terms(D + 4, D + 3, A + 2, X + 5);
            cyc_a = terms(A + 2, A + 5);
            cyc_b = terms(A + 2, X + 5);
            break;
        default:
            sqr_a = terms(A, A + 1, A + 2, Z);
            sqr_b = terms(D + 5, D + 4, D + 3, Z);
            cyc_a = terms(A + 1, Z);
            cyc_b = terms(D + 4, Z);
            break;
        }
        if (m == 0) st(kSlZero, Fq2::zero());
        __syncwarp();
    }

    __device__ __forceinline__ void st(int slot, const Fq2 &v) const
    {
        if (!live) return;
        uint4 *p = s + slot * kSlotChunks;
        p[0] = make_uint4(v.c0.v[0], v.c0.v[1], v.c0.v[2], v.c0.v[3]);
        p[1] = make_uint4(v.c0.v[4], v.c0.v[5], v.c0.v[6], v.c0.v[7]);
        p[2] = make_uint4(v.c1.v[0], v.c1.v[1], v.c1.v[2], v.c1.v[3]);
        p[3] = make_uint4(v.c1.v[4], v.c1.v[5], v.c1.v[6], v.c1.v[7]);
    }
    __device__ __forceinline__ Fq2 ld(int slot) const
    {
        Fq2 v;
        load_half(s + slot * kSlotChunks, v.c0.v);
        load_half(s + slot * kSlotChunks + 2, v.c1.v);
        return v;
    }
    // one product per lane: byte m of a and of b names the lane's operands
    __device__ __forceinline__ Fq2 level(uint64_t a, uint64_t b) const
    {
        const Fq2 r = lane_dot(s, 1, (a >> (8 * m)) & 255u, (b >> (8 * m)) & 255u);
        __syncwarp(); // every lane has read its operands
        return r;
    }

    // f g
    __device__ __noinline__ Fq2 mul(Fq2 f, Fq2 g) const
    {
        st(kSlA + m, f);
        st(kSlB + m, g);
        st(kSlXB + m, mul_xi(g));
        __syncwarp();
        uint64_t ta = 0, tb = 0;
#pragma unroll
        for (int i = 0; i < kPairLanes; ++i) {
            ta |= uint64_t(kSlA + i) << (8 * i);
            tb |= uint64_t(i <= m ? kSlB + m - i : kSlXB + m - i + kPairLanes) << (8 * i);
        }
        const Fq2 r = lane_dot(s, kPairLanes, ta, tb);
        __syncwarp();
        return r;
    }
    __device__ __forceinline__ void st_square(const Fq2 &f) const
    {
        const Fq2 x = mul_xi(f);
        st(kSlA + m, f);
        st(kSlXA + m, x);
        st(kSlB + m, dbl(f));
        st(kSlXB + m, dbl(x));
        __syncwarp();
    }
    __device__ __noinline__ Fq2 square(Fq2 f) const
    {
        st_square(f);
        const Fq2 r = lane_dot(s, 4, sqr_a, sqr_b);
        __syncwarp();
        return r;
    }
    // f^2 for f in the cyclotomic subgroup: 3 d - 2 a (even m) or 3 d + 2 a (odd m)
    __device__ __noinline__ Fq2 cyclotomic_square(Fq2 f) const
    {
        st_square(f);
        const Fq2 d = lane_dot(s, 2, cyc_a, cyc_b);
        __syncwarp();
        const Fq2 t = m & 1 ? d + f : d - f;
        return dbl(t) + d;
    }
    // f (c0 + a w + b w^3), the line in slots line .. line + 4
    __device__ __noinline__ Fq2 mul_line(Fq2 f, int line) const
    {
        st(kSlA + m, f);
        __syncwarp();
        const uint64_t ta = terms(kSlA + m, kSlA + (m + 5) % 6, kSlA + (m + 3) % 6);
        const uint64_t tb = terms(line, line + (m >= 1 ? 1 : 3), line + (m >= 3 ? 2 : 4));
        const Fq2 r = lane_dot(s, 3, ta, tb);
        __syncwarp();
        return r;
    }
    // conjugate: f(-w)
    __device__ __forceinline__ Fq2 conjugate(const Fq2 &f) const { return m & 1 ? neg(f) : f; }
    __device__ __forceinline__ Fq2 frobenius_map(const Fq2 &f, int k) const { return frob_coeff(f, k, m); }

    // conj(f) / f = conj(f)^2 / N with N = f conj(f) in Fq6 (coefficients c0, c1, c2 of 1, w^2,
    // w^4): 1 / N = (t0, t1, t2) / d with t0 = c0^2 - xi c1 c2, t1 = xi c2^2 - c0 c1,
    // t2 = c1^2 - c0 c2 and d = c0 t0 + xi (c2 t1 + c1 t2)
    __device__ __noinline__ Fq2 conj_over(Fq2 f) const
    {
        const Fq2 cf = conjugate(f);
        const Fq2 n = mul(f, cf);
        // slots: N's coefficients at A, xi N at XA, -N at B, -xi N at XB
        const Fq2 xn = mul_xi(n);
        st(kSlA + m, n);
        st(kSlXA + m, xn);
        st(kSlB + m, neg(n));
        st(kSlXB + m, neg(xn));
        __syncwarp();
        // lanes 0, 1, 2: t0, t1, t2
        const int c0 = 0, c1 = 2, c2 = 4;
        const uint64_t ta = m == 0 ? terms(kSlA + c0, kSlA + c1)
                            : m == 1 ? terms(kSlA + c2, kSlA + c0) : terms(kSlA + c1, kSlA + c0);
        const uint64_t tb = m == 0 ? terms(kSlA + c0, kSlXB + c2)
                            : m == 1 ? terms(kSlXA + c2, kSlB + c1) : terms(kSlA + c1, kSlB + c2);
        const Fq2 t = lane_dot(s, 2, ta, tb);
        __syncwarp();
        if (m < 3) st(kSlB + m, t);
        __syncwarp();
        // d, in every lane
        const Fq2 d = lane_dot(s, 3, terms(kSlA + c0, kSlXA + c2, kSlXA + c1), terms(kSlB, kSlB + 1, kSlB + 2));
        __syncwarp();
        st(kSlXB, inverse(d));
        __syncwarp();
        // coefficient 2 j of 1 / N is t_j / d
        Fq2 g = lane_dot(s, 1, kSlB + (m >> 1), kSlXB);
        __syncwarp();
        if (m & 1) g = Fq2::zero();
        return mul(mul(cf, cf), g);
    }

    // x^-z, x in the cyclotomic subgroup (inverses are conjugates), by z's signed digits: 13
    // products by x, x^3, x^5, x^7 or their inverses and 3 for these powers, against 27 for
    // the bits of z (4,096 verifications 5.29 -> 5.10 ms); the powers wait in the line slots
    __device__ __noinline__ Fq2 power_neg_z(Fq2 x) const
    {
        const Fq2 x2 = cyclotomic_square(x);
        Fq2 y = x;
        for (int k = 0; k < 3; ++k) { // x^3, x^5, x^7
            y = mul(x2, y);
            st(kSlLine + 6 * k + m, y);
        }
        Fq2 r = x; // digit 62 is 1
        for (int b = 61; b >= 0; --b) {
            r = cyclotomic_square(r);
            const int d = z_digit(b);
            if (d == 0) continue;
            const int k = (d < 0 ? -d : d) >> 1; // |d| = 2 k + 1
            y = k == 0 ? x : ld(kSlLine + 6 * (k - 1) + m);
            r = mul(r, d < 0 ? conjugate(y) : y);
        }
        return conjugate(r);
    }

    // f^((q^6 - 1)(q^2 + 1)) (the easy part), then libff's last chunk
    // (alt_bn128_pairing.cpp:152-224, Fuentes-Castaneda et al.): the same addition chain, so
    // the result is libff's GT value elt^(2z(6z^2 + 3z + 1)(q^4 - q^2 + 1)/r)
    __device__ __noinline__ Fq2 final_power(Fq2 f) const
    {
        const Fq2 c = conj_over(f);
        const Fq2 elt = mul(frobenius_map(c, 2), c);
        const Fq2 A = power_neg_z(elt);
        const Fq2 B = cyclotomic_square(A);
        const Fq2 C = cyclotomic_square(B);
        const Fq2 D = mul(C, B);
        const Fq2 E = power_neg_z(D);
        const Fq2 F = cyclotomic_square(E);
        const Fq2 G = power_neg_z(F);
        const Fq2 K = mul(mul(conjugate(G), E), conjugate(D)); // 12z^3 + 6z^2 + 6z
        const Fq2 L = mul(K, B);                               // 12z^3 + 6z^2 + 4z
        const Fq2 N = mul(mul(K, E), elt);                     // 12z^3 + 12z^2 + 6z + 1
        const Fq2 R = mul(frobenius_map(K, 2), mul(frobenius_map(L, 1), N));
        return mul(frobenius_map(mul(conjugate(elt), L), 3), R);
    }

    // The lines of pairs 1 and 2 at a step come from tables (slope lam, c), lanes 2 and 3
    // fetch them; a pair that is off has the line 1.
    struct Fixed {
        const AteLine *lines[2];
        bool on[2];
    };
    __device__ __forceinline__ void fetch(const Fixed &fx, int step) const
    {
        if (m == 2 || m == 3) {
            const int j = m - 2, line = kSlLine + 5 * (j + 1);
            AteLine l{Fq2::zero(), Fq2::zero()};
            if (fx.on[j]) l = fx.lines[j][step];
            st(line + 1, l.lam);
            st(line + 2, l.c);
        }
    }
    // after the first level: lane 2 and 3 hold a = -lam xP, lane 4 pair 1's b (scaled)
    __device__ __forceinline__ void st_fixed(const Fq2 &d) const
    {
        if (m == 2 || m == 3) {
            const int line = kSlLine + 5 * (m - 1);
            st(line + 1, d);
            st(line + 3, mul_xi(d));
            if (m == 3) st(line + 4, mul_xi(ld(line + 2)));
        }
        if (m == 4) {
            const int line = kSlLine + 5;
            st(line + 2, d);
            st(line + 4, mul_xi(d));
        }
    }
    // pair 0's line is 1 while the pair is off
    __device__ __forceinline__ void st_line0(bool on, int part, const Fq2 &v) const
    {
        const Fq2 w = on ? v : part == 0 ? Fq2::one() : Fq2::zero();
        st(kSlLine + part, w);
        if (part) st(kSlLine + part + 2, mul_xi(w));
    }

    // Pair 0's point runs T in homogeneous coordinates (x = X/Z, y = Y/Z), so that no step
    // inverts; its lines are the affine ones times an Fq2 factor (2YZ^2 for a doubling,
    // xQ Z - X for an addition) that the final exponentiation removes.
    //
    // Line through T and itself, T <- 2T: with a = 3X^2, b = 2YZ (slope a/b),
    // 2T = ((a^2 Z - 2X b^2) b, a (3X b^2 - a^2 Z) - Y b^3, b^3 Z).  Four levels of one
    // product per lane; lanes 2-4 of the first one compute the other pairs' lines.
    __device__ __noinline__ void double_step(const Fixed &fx, int step, bool on0, Fq scale1) const
    {
        constexpr int T = kSlT, Z0 = kSlZero;
        fetch(fx, step);
        if (m == 4) st(kSlScale1, Fq2{scale1, Fq::zero()});
        __syncwarp();
        Fq2 d = level(lane_bytes(kSlX, kSlY, kSlLine + 6, kSlLine + 11, kSlLine + 7, Z0),
                      lane_bytes(kSlX, kSlZ, kSlNegPx1, kSlNegPx2, kSlScale1, Z0));
        if (m == 0) st(T, dbl(d) + d);  // a = 3 X^2
        if (m == 1) st(T + 1, dbl(d));  // b = 2 Y Z
        st_fixed(d);
        __syncwarp();
        // b^2, a^2, a X, Y b, b Z, a Z
        d = level(lane_bytes(T + 1, T, T, kSlY, T + 1, T), lane_bytes(T + 1, T, kSlX, T + 1, kSlZ, kSlZ));
        st(T + 2 + m, d);
        __syncwarp();
        // b^3, a^2 Z, X b^2, c0 = b Z yP, line a = -a Z xP; lane 5: line b = a X - Y b
        d = level(lane_bytes(T + 2, T + 3, kSlX, T + 6, T + 7, Z0), lane_bytes(T + 1, kSlZ, T + 2, kSlPy, kSlNegPx, Z0));
        if (m < 3) st(T + 8 + m, d);
        if (m == 3) st_line0(on0, 0, d);
        if (m == 4) st_line0(on0, 1, d);
        if (m == 5) st_line0(on0, 2, ld(T + 4) - ld(T + 5));
        __syncwarp();
        if (m < 2) {
            const Fq2 a2z = ld(T + 9), xb2 = ld(T + 10), x2 = dbl(xb2);
            st(T + 2 + m, m == 0 ? a2z - x2 : x2 + xb2 - a2z);
        }
        __syncwarp();
        // X', a (3 X b^2 - a^2 Z), Y b^3, Z'
        d = level(lane_bytes(T + 2, T, kSlY, T + 8, Z0, Z0), lane_bytes(T + 1, T + 3, T + 8, kSlZ, Z0, Z0));
        if (m == 0) st(kSlX, d);
        if (m == 2) st(T + 4, d);
        if (m == 3) st(kSlZ, d);
        __syncwarp();
        if (m == 1) st(kSlY, d - ld(T + 4));
        __syncwarp();
    }

    // Line through T and the affine Q in kSlQx, kSlQy, T <- T + Q: with n = yQ Z - Y,
    // d = xQ Z - X (slope n/d), T + Q = ((n^2 Z - (X + xQ Z) d^2) d,
    // n ((2X + xQ Z) d^2 - n^2 Z) - Y d^3, d^3 Z)
    __device__ __noinline__ void add_step(const Fixed &fx, int step, bool on0, Fq scale1) const
    {
        constexpr int T = kSlT, Z0 = kSlZero;
        fetch(fx, step);
        if (m == 4) st(kSlScale1, Fq2{scale1, Fq::zero()});
        __syncwarp();
        Fq2 d = level(lane_bytes(kSlQy, kSlQx, kSlLine + 6, kSlLine + 11, kSlLine + 7, Z0),
                      lane_bytes(kSlZ, kSlZ, kSlNegPx1, kSlNegPx2, kSlScale1, Z0));
        if (m == 0) st(T, d - ld(kSlY)); // n = yQ Z - Y
        if (m == 1) {
            const Fq2 x = ld(kSlX), e = x + d;
            st(T + 1, d - x);            // d = xQ Z - X
            st(T + 2, e);                // X + xQ Z
            st(T + 3, e + x);            // 2 X + xQ Z
        }
        st_fixed(d);
        __syncwarp();
        // d^2, n^2, n xQ, yQ d, c0 = d yP, line a = -n xP
        d = level(lane_bytes(T + 1, T, T, kSlQy, T + 1, T),
                  lane_bytes(T + 1, T, kSlQx, T + 1, kSlPy, kSlNegPx));
        if (m < 4) st(T + 4 + m, d);
        if (m == 4) st_line0(on0, 0, d);
        if (m == 5) st_line0(on0, 1, d);
        __syncwarp();
        // d^3, n^2 Z, (X + xQ Z) d^2, (2 X + xQ Z) d^2; lane 5: line b = n xQ - yQ d
        d = level(lane_bytes(T + 4, T + 5, T + 2, T + 3, Z0, Z0), lane_bytes(T + 1, kSlZ, T + 4, T + 4, Z0, Z0));
        if (m < 4) st(T + 8 + m, d);
        if (m == 5) st_line0(on0, 2, ld(T + 6) - ld(T + 7));
        __syncwarp();
        if (m == 0) st(T + 4, ld(T + 9) - ld(T + 10));
        if (m == 1) st(T + 5, ld(T + 11) - ld(T + 9));
        __syncwarp();
        d = level(lane_bytes(T + 4, T, kSlY, T + 8, Z0, Z0), lane_bytes(T + 1, T + 5, T + 8, kSlZ, Z0, Z0));
        if (m == 0) st(kSlX, d);
        if (m == 2) st(T + 6, d);
        if (m == 3) st(kSlZ, d);
        __syncwarp();
        if (m == 1) st(kSlY, d - ld(T + 6));
        __syncwarp();
    }

    // The product of the three Miller loops: pair 0 is (P, Q) with lines of Q computed here,
    // pairs 1 and 2 have tabulated lines; `fixed` false leaves pairs 1 and 2 out.  Q's
    // coordinates are in kSlQx, kSlQy, the P in kSlNegPx .. kSlNegPx2 and the c0 of pairs
    // 1 and 2 in their line slots.
    __device__ __noinline__ Fq2 miller(const Fixed &fx, bool on0, bool fixed, Fq scale1) const
    {
        const Affine<Fq2> q{ld(kSlQx), ld(kSlQy)};
        if (m == 0) {
            st(kSlX, q.x);
            st(kSlY, q.y);
            st(kSlZ, Fq2::one());
        }
        __syncwarp();
        Fq2 f = m == 0 ? Fq2::one() : Fq2::zero();
        auto lines = [&] {
            f = mul_line(f, kSlLine);
            if (fixed) {
                f = mul_line(f, kSlLine + 5);
                f = mul_line(f, kSlLine + 10);
            }
        };
        int step = 0;
        for (int bit = kAteTopBit - 1; bit >= 0; --bit) {
            f = square(f);
            double_step(fx, step++, on0, scale1);
            lines();
            if (ate_bit(bit)) {
                add_step(fx, step++, on0, scale1);
                lines();
            }
        }
        for (int k = 0; k < 2; ++k) {
            const Affine<Fq2> e = k == 0 ? twist_frobenius(q) : twist_neg_frobenius2(q);
            if (m == 0) {
                st(kSlQx, e.x);
                st(kSlQy, e.y);
            }
            __syncwarp();
            add_step(fx, step++, on0, scale1);
            lines();
        }
        return f;
    }

    // index of coefficient m among the six Fq2 of an Fq12 in memory: w^m = v^(m / 2) w^(m % 2)
    __device__ __forceinline__ int tower_index() const { return (m & 1) * 3 + (m >> 1); }
};

} // namespace nkr
