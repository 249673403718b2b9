// BN254 base field Fq and scalar field Fr on sm_100a.
//
// Representation: 8 x 32-bit little-endian limbs in Montgomery form
// (R = 2^256), in memory always fully reduced (< modulus); kernels compute in Fp, fully
// reduced as well, or on values below twice the modulus (FpL, Fq2M).  The byte image is
// identical to libff's Fp_model<4, modulus>::mont_repr on x86-64, so device buffers are
// bit-for-bit the reference's host vectors (reference: libff
// algebra/fields/fp.hpp:40-42, CUDA mont_t layout operators/cuda/include/fields/
// mont_t.cuh:45).
//
// Multiplication is row-wise Montgomery with the running value split into an even
// and an odd accumulator (mont_mul below).  Because p < 2^254, the running value
// stays below 2^288 and 9 words suffice.
#pragma once

#include <cstdint>

namespace nkr {

struct FqParams {
    static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du,
                              P3 = 0x97816a91u, P4 = 0x8181585du, P5 = 0xb85045b6u,
                              P6 = 0xe131a029u, P7 = 0x30644e72u;
    static constexpr uint32_t INV = 0xe4866389u; // -p^-1 mod 2^32
    static constexpr uint32_t O0 = 0xc58f0d9du, O1 = 0xd35d438du, O2 = 0xf5c70b3du, O3 = 0x0a78eb28u, O4 = 0x7879462cu, O5 = 0x666ea36fu, O6 = 0x9a07df2fu, O7 = 0x0e0a77c1u;
    static constexpr uint32_t Q0 = 0x538afa89u, Q1 = 0xf32cfc5bu, Q2 = 0xd44501fbu, Q3 = 0xb5e71911u, Q4 = 0x0a417ff6u, Q5 = 0x47ab1effu, Q6 = 0xcab8351fu, Q7 = 0x06d89f71u;
};

struct FrParams {
    static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u,
                              P3 = 0x2833e848u, P4 = 0x8181585du, P5 = 0xb85045b6u,
                              P6 = 0xe131a029u, P7 = 0x30644e72u;
    static constexpr uint32_t INV = 0xefffffffu;
    static constexpr uint32_t O0 = 0x4ffffffbu, O1 = 0xac96341cu, O2 = 0x9f60cd29u, O3 = 0x36fc7695u, O4 = 0x7879462eu, O5 = 0x666ea36fu, O6 = 0x9a07df2fu, O7 = 0x0e0a77c1u;
    static constexpr uint32_t Q0 = 0xae216da7u, Q1 = 0x1bb8e645u, Q2 = 0xe35c59e3u, Q3 = 0x53fe3ab1u, Q4 = 0x53bb8085u, Q5 = 0x8c49833du, Q6 = 0x7f4e44a5u, Q7 = 0x0216d0b1u;
};

template <class P>
struct alignas(32) Fp {
    uint32_t v[8];

    __device__ __forceinline__ static Fp zero()
    {
        Fp r;
#pragma unroll
        for (int i = 0; i < 8; ++i) r.v[i] = 0;
        return r;
    }
    __device__ __forceinline__ static Fp one()
    {
        return {{P::O0, P::O1, P::O2, P::O3, P::O4, P::O5, P::O6, P::O7}};
    }
    __device__ __forceinline__ static Fp r2()
    {
        return {{P::Q0, P::Q1, P::Q2, P::Q3, P::Q4, P::Q5, P::Q6, P::Q7}};
    }
    __device__ __forceinline__ bool is_zero() const
    {
        uint32_t x = v[0];
#pragma unroll
        for (int i = 1; i < 8; ++i) x |= v[i];
        return x == 0;
    }
    __device__ __forceinline__ bool operator==(const Fp &o) const
    {
        uint32_t x = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) x |= v[i] ^ o.v[i];
        return x == 0;
    }
    __device__ __forceinline__ bool operator!=(const Fp &o) const { return !(*this == o); }
};

using Fq = Fp<FqParams>;
using Fr = Fp<FrParams>;

// ---------------------------------------------------------------------------
// conditional subtraction of the modulus: r = (t >= p) ? t - p : t
// ---------------------------------------------------------------------------
template <class P>
__device__ __forceinline__ void reduce_once(uint32_t *t)
{
    uint32_t s0, s1, s2, s3, s4, s5, s6, s7, br;
    asm("sub.cc.u32  %0, %9,  %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(s0), "=r"(s1), "=r"(s2), "=r"(s3), "=r"(s4), "=r"(s5), "=r"(s6), "=r"(s7),
          "=r"(br)
        : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]),
          "r"(t[7]), "n"(P::P0), "n"(P::P1), "n"(P::P2), "n"(P::P3), "n"(P::P4), "n"(P::P5),
          "n"(P::P6), "n"(P::P7));
    // br == 0xffffffff when t < p (keep t), 0 when t >= p (take t - p)
    const bool keep = br != 0;
    t[0] = keep ? t[0] : s0;
    t[1] = keep ? t[1] : s1;
    t[2] = keep ? t[2] : s2;
    t[3] = keep ? t[3] : s3;
    t[4] = keep ? t[4] : s4;
    t[5] = keep ? t[5] : s5;
    t[6] = keep ? t[6] : s6;
    t[7] = keep ? t[7] : s7;
}

template <class P>
__device__ __forceinline__ Fp<P> operator+(const Fp<P> &a, const Fp<P> &b)
{
    Fp<P> r;
    asm("add.cc.u32  %0, %8,  %16;\n\t"
        "addc.cc.u32 %1, %9,  %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
          "=r"(r.v[6]), "=r"(r.v[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]),
          "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    reduce_once<P>(r.v);
    return r;
}

template <class P>
__device__ __forceinline__ Fp<P> operator-(const Fp<P> &a, const Fp<P> &b)
{
    Fp<P> r;
    uint32_t br;
    asm("sub.cc.u32  %0, %9,  %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
          "=r"(r.v[6]), "=r"(r.v[7]), "=r"(br)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]),
          "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    // on borrow add p back (br is an all-ones mask)
    asm("add.cc.u32  %0, %0, %8;\n\t"
        "addc.cc.u32 %1, %1, %9;\n\t"
        "addc.cc.u32 %2, %2, %10;\n\t"
        "addc.cc.u32 %3, %3, %11;\n\t"
        "addc.cc.u32 %4, %4, %12;\n\t"
        "addc.cc.u32 %5, %5, %13;\n\t"
        "addc.cc.u32 %6, %6, %14;\n\t"
        "addc.u32    %7, %7, %15;"
        : "+&r"(r.v[0]), "+&r"(r.v[1]), "+&r"(r.v[2]), "+&r"(r.v[3]), "+&r"(r.v[4]), "+&r"(r.v[5]),
          "+&r"(r.v[6]), "+&r"(r.v[7])
        : "r"(P::P0 & br), "r"(P::P1 & br), "r"(P::P2 & br), "r"(P::P3 & br), "r"(P::P4 & br),
          "r"(P::P5 & br), "r"(P::P6 & br), "r"(P::P7 & br));
    return r;
}

template <class P>
__device__ __forceinline__ Fp<P> neg(const Fp<P> &a)
{
    return Fp<P>::zero() - a;
}

template <class P>
__device__ __forceinline__ Fp<P> dbl(const Fp<P> &a)
{
    return a + a;
}

// One CIOS round: t[0..8] += a * bi; m = t0 * inv; t += m * p; t >>= 32.
#define NKR_CIOS_ROUND(bi)                                                                     \
    asm("mad.lo.cc.u32  %0, %9,  %17, %0;\n\t"                                                 \
        "madc.lo.cc.u32 %1, %10, %17, %1;\n\t"                                                 \
        "madc.lo.cc.u32 %2, %11, %17, %2;\n\t"                                                 \
        "madc.lo.cc.u32 %3, %12, %17, %3;\n\t"                                                 \
        "madc.lo.cc.u32 %4, %13, %17, %4;\n\t"                                                 \
        "madc.lo.cc.u32 %5, %14, %17, %5;\n\t"                                                 \
        "madc.lo.cc.u32 %6, %15, %17, %6;\n\t"                                                 \
        "madc.lo.cc.u32 %7, %16, %17, %7;\n\t"                                                 \
        "addc.u32       %8, %8, 0;\n\t"                                                        \
        "mad.hi.cc.u32  %1, %9,  %17, %1;\n\t"                                                 \
        "madc.hi.cc.u32 %2, %10, %17, %2;\n\t"                                                 \
        "madc.hi.cc.u32 %3, %11, %17, %3;\n\t"                                                 \
        "madc.hi.cc.u32 %4, %12, %17, %4;\n\t"                                                 \
        "madc.hi.cc.u32 %5, %13, %17, %5;\n\t"                                                 \
        "madc.hi.cc.u32 %6, %14, %17, %6;\n\t"                                                 \
        "madc.hi.cc.u32 %7, %15, %17, %7;\n\t"                                                 \
        "madc.hi.u32    %8, %16, %17, %8;"                                                     \
        : "+&r"(t0), "+&r"(t1), "+&r"(t2), "+&r"(t3), "+&r"(t4), "+&r"(t5), "+&r"(t6), "+&r"(t7),      \
          "+&r"(t8)                                                                             \
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),        \
          "r"(a.v[6]), "r"(a.v[7]), "r"(bi));                                                  \
    {                                                                                          \
        const uint32_t m = t0 * P::INV;                                                        \
        asm("mad.lo.cc.u32  %0, %9, %10, %0;\n\t"                                              \
            "madc.lo.cc.u32 %1, %9, %11, %1;\n\t"                                              \
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"                                              \
            "madc.lo.cc.u32 %3, %9, %13, %3;\n\t"                                              \
            "madc.lo.cc.u32 %4, %9, %14, %4;\n\t"                                              \
            "madc.lo.cc.u32 %5, %9, %15, %5;\n\t"                                              \
            "madc.lo.cc.u32 %6, %9, %16, %6;\n\t"                                              \
            "madc.lo.cc.u32 %7, %9, %17, %7;\n\t"                                              \
            "addc.u32       %8, %8, 0;\n\t"                                                    \
            "mad.hi.cc.u32  %1, %9, %10, %1;\n\t"                                              \
            "madc.hi.cc.u32 %2, %9, %11, %2;\n\t"                                              \
            "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"                                              \
            "madc.hi.cc.u32 %4, %9, %13, %4;\n\t"                                              \
            "madc.hi.cc.u32 %5, %9, %14, %5;\n\t"                                              \
            "madc.hi.cc.u32 %6, %9, %15, %6;\n\t"                                              \
            "madc.hi.cc.u32 %7, %9, %16, %7;\n\t"                                              \
            "madc.hi.u32    %8, %9, %17, %8;"                                                  \
            : "+&r"(t0), "+&r"(t1), "+&r"(t2), "+&r"(t3), "+&r"(t4), "+&r"(t5), "+&r"(t6), "+&r"(t7),  \
              "+&r"(t8)                                                                         \
            : "r"(m), "n"(P::P0), "n"(P::P1), "n"(P::P2), "n"(P::P3), "n"(P::P4), "n"(P::P5),  \
              "n"(P::P6), "n"(P::P7));                                                         \
    }                                                                                          \
    t0 = t1;                                                                                   \
    t1 = t2;                                                                                   \
    t2 = t3;                                                                                   \
    t3 = t4;                                                                                   \
    t4 = t5;                                                                                   \
    t5 = t6;                                                                                   \
    t6 = t7;                                                                                   \
    t7 = t8;                                                                                   \
    t8 = 0;

// Translation units whose kernels chain many products (curve arithmetic) define
// NKR_FIELD_MUL_OUTLINE before including this header: the product body then
// exists once per kernel instead of once per call site, which keeps the hot
// loop inside the instruction cache (inlined, one XYZZ addition is several
// thousand instructions).  Elementwise kernels keep it inlined.
// NKR_MUL_ATTR_FN is the same for non-template functions, which also need
// `inline` to be defined in every translation unit that includes the header.
#ifdef NKR_FIELD_MUL_OUTLINE
#define NKR_MUL_ATTR __noinline__
#define NKR_MUL_ATTR_FN inline __noinline__
#else
#define NKR_MUL_ATTR __forceinline__
#define NKR_MUL_ATTR_FN __forceinline__
#endif

template <class P>
__device__ __forceinline__ uint32_t mod_word(int j)
{
    switch (j) {
    case 0: return P::P0;
    case 1: return P::P1;
    case 2: return P::P2;
    case 3: return P::P3;
    case 4: return P::P4;
    case 5: return P::P5;
    case 6: return P::P6;
    default: return P::P7;
    }
}

// ---------------------------------------------------------------------------
// The Montgomery product.  A 32 x 32 -> 64-bit multiply-add with carry in and out
// is one instruction (a mad.lo / madc.hi pair on two adjacent words), but only
// when its 64-bit addend sits in one aligned word pair.  Row i of a x b has eight
// partial products at word offsets 0..7: those of the even words of a go to the
// accumulator E (pairs at offsets 0, 2, 4, 6), those of the odd words to O (pairs at
// 1, 3, 5, 7), so every row is four multiply-adds in one carry chain per
// accumulator, with no 64-bit addition beside them; m p is added the same way.
// Shifting the running value down one word turns O into the next row's E and E,
// less its two lowest words, into its O; the word E[1] left over enters the first
// multiply-add of the next row as its addend, which cannot overflow.
//
// Bound: the multiply pipe, which takes a wide multiply-add every 4 cycles per warp
// (measured 25-32 lanes per SM and cycle): 128 of them are 512 cycles.  Against the
// form it replaces (one 64-bit sum per partial product, 219 additions on the ALU
// pipe and 130 more on the multiply pipe): 43.5 -> 63.7e9 products/s in registers,
// 579 -> 438 ns for one product after another with one warp per scheduler (B200,
// 1965 MHz).
// ---------------------------------------------------------------------------

// (x0..x7) += (a0, a2, a4, a6) b at word offsets 0, 2, 4, 6; c += carry out
__device__ __forceinline__ void eo_mad(uint32_t *x, uint32_t &c, uint32_t a0, uint32_t a2, uint32_t a4,
                                       uint32_t a6, uint32_t b)
{
    asm("mad.lo.cc.u32  %0, %9,  %13, %0;\n\t"
        "madc.hi.cc.u32 %1, %9,  %13, %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
        "addc.u32       %8, %8, 0;"
        : "+&r"(x[0]), "+&r"(x[1]), "+&r"(x[2]), "+&r"(x[3]), "+&r"(x[4]), "+&r"(x[5]), "+&r"(x[6]),
          "+&r"(x[7]), "+&r"(c)
        : "r"(a0), "r"(a2), "r"(a4), "r"(a6), "r"(b));
}

// the same where the sum is known to fit eight words
__device__ __forceinline__ void eo_mad_fit(uint32_t *x, uint32_t a0, uint32_t a2, uint32_t a4, uint32_t a6,
                                           uint32_t b)
{
    asm("mad.lo.cc.u32  %0, %8,  %12, %0;\n\t"
        "madc.hi.cc.u32 %1, %8,  %12, %1;\n\t"
        "madc.lo.cc.u32 %2, %9,  %12, %2;\n\t"
        "madc.hi.cc.u32 %3, %9,  %12, %3;\n\t"
        "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
        "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
        "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
        "madc.hi.u32    %7, %11, %12, %7;"
        : "+&r"(x[0]), "+&r"(x[1]), "+&r"(x[2]), "+&r"(x[3]), "+&r"(x[4]), "+&r"(x[5]), "+&r"(x[6]), "+&r"(x[7])
        : "r"(a0), "r"(a2), "r"(a4), "r"(a6), "r"(b));
}

// (x0..x7) += (a0, a2, a4, a6) b + w with one word w; c = carry out
__device__ __forceinline__ void eo_mad_word(uint32_t *x, uint32_t &c, uint32_t w, uint32_t a0, uint32_t a2,
                                            uint32_t a4, uint32_t a6, uint32_t b)
{
    asm("{\n\t"
        ".reg .u32 l, h;\n\t"
        "mad.lo.cc.u32  l,  %9,  %13, %14;\n\t"
        "madc.hi.u32    h,  %9,  %13, 0;\n\t"
        "add.cc.u32     %0, %0,  l;\n\t"
        "addc.cc.u32    %1, %1,  h;\n\t"
        "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
        "addc.u32       %8, 0, 0;\n\t"
        "}"
        : "+&r"(x[0]), "+&r"(x[1]), "+&r"(x[2]), "+&r"(x[3]), "+&r"(x[4]), "+&r"(x[5]), "+&r"(x[6]),
          "+&r"(x[7]), "=r"(c)
        : "r"(a0), "r"(a2), "r"(a4), "r"(a6), "r"(b), "r"(w));
}

// r = x + y on eight words
__device__ __forceinline__ void add_words(uint32_t *r, const uint32_t *x, const uint32_t *y)
{
    asm("add.cc.u32  %0, %8,  %16;\n\t"
        "addc.cc.u32 %1, %9,  %17;\n\t"
        "addc.cc.u32 %2, %10, %18;\n\t"
        "addc.cc.u32 %3, %11, %19;\n\t"
        "addc.cc.u32 %4, %12, %20;\n\t"
        "addc.cc.u32 %5, %13, %21;\n\t"
        "addc.cc.u32 %6, %14, %22;\n\t"
        "addc.u32    %7, %15, %23;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]),
          "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
}

// r = x + y + c on eight words, c = carry out
__device__ __forceinline__ void add_words_carry(uint32_t *r, const uint32_t *x, const uint32_t *y, uint32_t &c)
{
    asm("add.cc.u32  %8, %8,  0xffffffff;\n\t" // carry in
        "addc.cc.u32 %0, %9,  %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32    %8, 0, 0;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]),
          "=&r"(r[7]), "+&r"(c)
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]),
          "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
}

// r = x - y on 16 words (no borrow out); r may be x
__device__ __forceinline__ void sub_words16(uint32_t *r, const uint32_t *x, const uint32_t *y)
{
    uint32_t br;
    asm("sub.cc.u32  %0, %9,  %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]),
          "=&r"(r[7]), "=&r"(br)
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]),
          "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]), "r"(y[4]), "r"(y[5]), "r"(y[6]), "r"(y[7]));
    asm("sub.cc.u32  %8, 0,   %8;\n\t" // br is all ones on borrow: borrows again
        "subc.cc.u32 %0, %9,  %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.u32    %7, %16, %24;"
        : "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]),
          "=&r"(r[15]), "+&r"(br)
        : "r"(x[8]), "r"(x[9]), "r"(x[10]), "r"(x[11]), "r"(x[12]), "r"(x[13]), "r"(x[14]), "r"(x[15]),
          "r"(y[8]), "r"(y[9]), "r"(y[10]), "r"(y[11]), "r"(y[12]), "r"(y[13]), "r"(y[14]), "r"(y[15]));
}

// E[0..8], O[0..7] += m p with m = E[0] (-p^-1): word offset 0 becomes zero
template <class P>
__device__ __forceinline__ void eo_reduce_row(uint32_t *e, uint32_t *o)
{
    const uint32_t m = e[0] * P::INV;
    eo_mad_fit(o, P::P1, P::P3, P::P5, P::P7, m);
    eo_mad(e, e[8], P::P0, P::P2, P::P4, P::P6, m);
}

// a b 2^-256 mod p, below a b / 2^256 + p and not reduced further: for inputs
// below 2p the result is below 1.76 p.  The running value stays below
// 2^32 (a + p), within nine words for a < 2^256 - p; b may be any eight words (with a < p the
// result is below 2p then).  So a value that a caller hands in, which need not be reduced,
// goes second.
template <class P>
__device__ __forceinline__ void mont_mul(const uint32_t *a, const uint32_t *b, uint32_t *r)
{
    uint32_t e[9], o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint64_t x = uint64_t(a[2 * j]) * b[0], y = uint64_t(a[2 * j + 1]) * b[0];
        e[2 * j] = uint32_t(x);
        e[2 * j + 1] = uint32_t(x >> 32);
        o[2 * j] = uint32_t(y);
        o[2 * j + 1] = uint32_t(y >> 32);
    }
    e[8] = 0;
    eo_reduce_row<P>(e, o);
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        uint32_t ne[9], no[8];
        const uint32_t w = e[1];
#pragma unroll
        for (int j = 0; j < 8; ++j) ne[j] = o[j];
#pragma unroll
        for (int j = 0; j < 7; ++j) no[j] = e[j + 2];
        no[7] = 0;
        eo_mad_fit(no, a[1], a[3], a[5], a[7], b[i]);
        eo_mad_word(ne, ne[8], w, a[0], a[2], a[4], a[6], b[i]);
        eo_reduce_row<P>(ne, no);
#pragma unroll
        for (int j = 0; j < 9; ++j) e[j] = ne[j];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = no[j];
    }
    add_words(r, e + 1, o);
}

// Operands travel by value: an out-of-line call (NKR_FIELD_MUL_OUTLINE) then
// passes them in registers instead of through the thread's local-memory stack
// (measured 10% faster G2 MSMs than reference parameters).
template <class P>
__device__ NKR_MUL_ATTR Fp<P> operator*(Fp<P> a, Fp<P> b)
{
    Fp<P> r;
    mont_mul<P>(a.v, b.v, r.v);
    reduce_once<P>(r.v);
    return r;
}

// The same product with one accumulator and separate carry chains for the low and
// the high halves of every row (two half products each, none of which pairs up
// into a wide multiply-add); kept for comparison.
template <class P>
__device__ __forceinline__ Fp<P> mont_mul_cc(const Fp<P> &a, const Fp<P> &b)
{
    uint32_t t0 = 0, t1 = 0, t2 = 0, t3 = 0, t4 = 0, t5 = 0, t6 = 0, t7 = 0, t8 = 0;
    NKR_CIOS_ROUND(b.v[0])
    NKR_CIOS_ROUND(b.v[1])
    NKR_CIOS_ROUND(b.v[2])
    NKR_CIOS_ROUND(b.v[3])
    NKR_CIOS_ROUND(b.v[4])
    NKR_CIOS_ROUND(b.v[5])
    NKR_CIOS_ROUND(b.v[6])
    NKR_CIOS_ROUND(b.v[7])
    Fp<P> r;
    r.v[0] = t0;
    r.v[1] = t1;
    r.v[2] = t2;
    r.v[3] = t3;
    r.v[4] = t4;
    r.v[5] = t5;
    r.v[6] = t6;
    r.v[7] = t7;
    (void)t8;
    reduce_once<P>(r.v);
    return r;
}


// r = t[0..7] R^-1 mod p (R = 2^256), at most p: the rows of mont_mul without a product
template <class P>
__device__ __forceinline__ void redc_low(const uint32_t *t, uint32_t *r)
{
    uint32_t e[9], o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) e[j] = t[j], o[j] = 0;
    e[8] = 0;
    eo_reduce_row<P>(e, o);
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        uint32_t ne[9], no[8];
        const uint32_t w = e[1];
#pragma unroll
        for (int j = 0; j < 8; ++j) ne[j] = o[j];
#pragma unroll
        for (int j = 0; j < 7; ++j) no[j] = e[j + 2];
        no[7] = 0;
        const uint32_t m = (ne[0] + w) * P::INV;
        eo_mad_fit(no, P::P1, P::P3, P::P5, P::P7, m);
        eo_mad_word(ne, ne[8], w, P::P0, P::P2, P::P4, P::P6, m);
#pragma unroll
        for (int j = 0; j < 9; ++j) e[j] = ne[j];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = no[j];
    }
    add_words(r, e + 1, o);
}

// x += (a[0], a[2], ..) b, n words of a into adjacent word pairs of x, with the carry
// added to the word after them
__device__ __forceinline__ void mad_chain(uint32_t *x, const uint32_t *a, int n, uint32_t b)
{
    if (n == 4)
        eo_mad(x, x[8], a[0], a[2], a[4], a[6], b);
    else if (n == 3)
        asm("mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
            "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
            "addc.u32       %6, %6, 0;"
            : "+&r"(x[0]), "+&r"(x[1]), "+&r"(x[2]), "+&r"(x[3]), "+&r"(x[4]), "+&r"(x[5]), "+&r"(x[6])
            : "r"(a[0]), "r"(a[2]), "r"(a[4]), "r"(b));
    else if (n == 2)
        asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
            "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
            "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
            "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
            "addc.u32       %4, %4, 0;"
            : "+&r"(x[0]), "+&r"(x[1]), "+&r"(x[2]), "+&r"(x[3]), "+&r"(x[4])
            : "r"(a[0]), "r"(a[2]), "r"(b));
    else if (n == 1)
        asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
            "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
            "addc.u32       %2, %2, 0;"
            : "+&r"(x[0]), "+&r"(x[1]), "+&r"(x[2])
            : "r"(a[0]), "r"(b));
}

// t = 2 t + sum_i a_i^2 2^(64 i) on 16 words, 2 t < 2^512 and no carry out
__device__ __forceinline__ void double_add_squares(uint32_t *t, const uint32_t *a)
{
#pragma unroll
    for (int j = 15; j > 0; --j) t[j] = __funnelshift_l(t[j - 1], t[j], 1);
    t[0] <<= 1;
    uint32_t c = 0;
    asm("mad.lo.cc.u32  %0, %9,  %9,  %0;\n\t"
        "madc.hi.cc.u32 %1, %9,  %9,  %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %10, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %10, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %11, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %11, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %12, %6;\n\t"
        "madc.hi.cc.u32 %7, %12, %12, %7;\n\t"
        "addc.u32       %8, 0, 0;"
        : "+&r"(t[0]), "+&r"(t[1]), "+&r"(t[2]), "+&r"(t[3]), "+&r"(t[4]), "+&r"(t[5]), "+&r"(t[6]), "+&r"(t[7]), "=r"(c)
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]));
    asm("add.cc.u32     %8, %8,  0xffffffff;\n\t" // carry in
        "madc.lo.cc.u32 %0, %9,  %9,  %0;\n\t"
        "madc.hi.cc.u32 %1, %9,  %9,  %1;\n\t"
        "madc.lo.cc.u32 %2, %10, %10, %2;\n\t"
        "madc.hi.cc.u32 %3, %10, %10, %3;\n\t"
        "madc.lo.cc.u32 %4, %11, %11, %4;\n\t"
        "madc.hi.cc.u32 %5, %11, %11, %5;\n\t"
        "madc.lo.cc.u32 %6, %12, %12, %6;\n\t"
        "madc.hi.u32    %7, %12, %12, %7;"
        : "+&r"(t[8]), "+&r"(t[9]), "+&r"(t[10]), "+&r"(t[11]), "+&r"(t[12]), "+&r"(t[13]), "+&r"(t[14]), "+&r"(t[15]),
          "+&r"(c)
        : "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
}

// a^2 2^-256 mod p, bounds as mont_mul: the 28 products of distinct words once, doubled,
// and 8 squares, then the reduction of the low half (100 wide multiply-adds instead of 128)
template <class P>
__device__ __forceinline__ void mont_sqr(const uint32_t *a, uint32_t *r)
{
    uint32_t e[16], o[16]; // o[k] holds word offset k + 1
#pragma unroll
    for (int j = 0; j < 16; ++j) e[j] = o[j] = 0;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        // a_i a_j, j > i: offsets i + j odd into o, even into e; chains from the lowest
        mad_chain(o + 2 * i, a + i + 1, (8 - i) / 2, a[i]);
        mad_chain(e + 2 * i + 2, a + i + 2, (7 - i) / 2, a[i]);
    }
    uint32_t t[16], c = 0;
    t[0] = 0;
    uint32_t hi[8];
    add_words_carry(t + 1, e + 1, o, c);
    uint32_t eh[8];
#pragma unroll
    for (int j = 0; j < 7; ++j) eh[j] = e[9 + j];
    eh[7] = 0;
    add_words_carry(hi, eh, o + 8, c);
#pragma unroll
    for (int j = 0; j < 7; ++j) t[9 + j] = hi[j];
    double_add_squares(t, a);
    uint32_t lo[8];
    redc_low<P>(t, lo);
    add_words(r, lo, t + 8);
}

template <class P>
__device__ NKR_MUL_ATTR Fp<P> sqr(Fp<P> a)
{
    Fp<P> r;
    mont_sqr<P>(a.v, r.v);
    reduce_once<P>(r.v);
    return r;
}

// Montgomery -> canonical integer (same limb layout); any eight words
template <class P>
__device__ __forceinline__ Fp<P> from_mont(const Fp<P> &a)
{
    Fp<P> one;
    one.v[0] = 1;
#pragma unroll
    for (int i = 1; i < 8; ++i) one.v[i] = 0;
    return a * one; // (one's single word keeps the running value within nine words)
}

// integer (any eight words) -> Montgomery
template <class P>
__device__ __forceinline__ Fp<P> to_mont(const Fp<P> &a)
{
    return Fp<P>::r2() * a;
}

// the value below p congruent to eight words that a caller handed in (2^256 < 6p).  Not a
// product by one: with its calls at the head of the verification kernel 4,096 proofs take
// 5.63 ms, with this loop 5.14 ms, as with no reduction at all.
template <class P>
__device__ __forceinline__ Fp<P> reduced(Fp<P> a)
{
#pragma unroll 1
    for (int i = 0; i < 5; ++i) reduce_once<P>(a.v);
    return a;
}

// a b where either of them may be any eight words and the other one is below p
template <class P>
__device__ __forceinline__ Fp<P> mul_any(Fp<P> a, const Fp<P> &b)
{
    reduce_once<P>(a.v); // below 2^256 - p
    return a * b;
}

// a^e for a small public exponent given as 8 limbs (left-to-right square-and-multiply)
template <class P>
__device__ Fp<P> pow_limbs(const Fp<P> &a, const uint32_t *e)
{
    Fp<P> acc = Fp<P>::one();
    for (int i = 255; i >= 0; --i) {
        acc = sqr(acc);
        if ((e[i >> 5] >> (i & 31)) & 1) acc = acc * a;
    }
    return acc;
}

// Fermat inverse: a^(p-2).  0 maps to 0.
template <class P>
__device__ Fp<P> inverse(const Fp<P> &a)
{
    const uint32_t e[8] = {P::P0 - 2u, P::P1, P::P2, P::P3, P::P4, P::P5, P::P6, P::P7};
    return pow_limbs(a, e);
}

// ---------------------------------------------------------------------------
// FpL: values in [0, 2p), the compute type of the G1 MSM (FqL) and of the transforms
// (FrL).  A product of two such values is below 1.76 p as it stands (mont_mul), so
// products skip the conditional subtraction; additions and subtractions work modulo 2p.
// Zero tests accept 0 and p.  Values are made canonical when they leave for memory
// (canon()).
// ---------------------------------------------------------------------------

// 2p as a parameter set: reduce_once and the subtraction of Fp on it work modulo 2p
template <class P>
struct TwoP {
    static constexpr uint32_t P0 = P::P0 << 1, P1 = P::P1 << 1 | P::P0 >> 31, P2 = P::P2 << 1 | P::P1 >> 31,
                              P3 = P::P3 << 1 | P::P2 >> 31, P4 = P::P4 << 1 | P::P3 >> 31,
                              P5 = P::P5 << 1 | P::P4 >> 31, P6 = P::P6 << 1 | P::P5 >> 31,
                              P7 = P::P7 << 1 | P::P6 >> 31;
};

// (a b + c d) 2^-256 mod p with one reduction: for inputs below 2p the running value stays
// below 2^32 (a + c + p) <= 2^32 5p < 2^288 and the result below 2.51 p; one conditional
// subtraction of 2p brings it below 2p (192 wide multiply-adds instead of 256)
template <class P>
__device__ __forceinline__ void mont_mul_add(const uint32_t *a, const uint32_t *b, const uint32_t *x,
                                             const uint32_t *y, uint32_t *r)
{
    uint32_t e[9], o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint64_t u = uint64_t(a[2 * j]) * b[0], w = uint64_t(a[2 * j + 1]) * b[0];
        e[2 * j] = uint32_t(u);
        e[2 * j + 1] = uint32_t(u >> 32);
        o[2 * j] = uint32_t(w);
        o[2 * j + 1] = uint32_t(w >> 32);
    }
    e[8] = 0;
    eo_mad_fit(o, x[1], x[3], x[5], x[7], y[0]);
    eo_mad(e, e[8], x[0], x[2], x[4], x[6], y[0]);
    eo_reduce_row<P>(e, o);
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        uint32_t ne[9], no[8];
        const uint32_t w = e[1];
#pragma unroll
        for (int j = 0; j < 8; ++j) ne[j] = o[j];
#pragma unroll
        for (int j = 0; j < 7; ++j) no[j] = e[j + 2];
        no[7] = 0;
        eo_mad_fit(no, a[1], a[3], a[5], a[7], b[i]);
        eo_mad_word(ne, ne[8], w, a[0], a[2], a[4], a[6], b[i]);
        eo_mad_fit(no, x[1], x[3], x[5], x[7], y[i]);
        eo_mad(ne, ne[8], x[0], x[2], x[4], x[6], y[i]);
        eo_reduce_row<P>(ne, no);
#pragma unroll
        for (int j = 0; j < 9; ++j) e[j] = ne[j];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = no[j];
    }
    add_words(r, e + 1, o);
}

template <class P>
struct alignas(32) FpL {
    uint32_t v[8];
    FpL() = default;
    __device__ __forceinline__ FpL(const Fp<P> &c)
    {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = c.v[j];
    }
    __device__ __forceinline__ static FpL zero() { return Fp<P>::zero(); }
    __device__ __forceinline__ static FpL one() { return Fp<P>::one(); }
    __device__ __forceinline__ bool is_zero() const // 0 or p
    {
        uint32_t x = 0, y = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x |= v[j];
            y |= v[j] ^ mod_word<P>(j);
        }
        return x == 0 || y == 0;
    }
    __device__ __forceinline__ Fp<P> canon() const
    {
        Fp<P> r;
#pragma unroll
        for (int j = 0; j < 8; ++j) r.v[j] = v[j];
        reduce_once<P>(r.v);
        return r;
    }
    __device__ __forceinline__ bool operator==(const FpL &o) const { return canon() == o.canon(); }
    __device__ __forceinline__ bool operator!=(const FpL &o) const { return !(*this == o); }
};
using FqL = FpL<FqParams>;
using FrL = FpL<FrParams>;

template <class P>
__device__ NKR_MUL_ATTR FpL<P> operator*(FpL<P> a, FpL<P> b)
{
    FpL<P> r;
    mont_mul<P>(a.v, b.v, r.v);
    return r;
}
template <class P>
__device__ NKR_MUL_ATTR FpL<P> sqr(FpL<P> a)
{
    FpL<P> r;
    mont_sqr<P>(a.v, r.v);
    return r;
}
// a b + c d
template <class P>
__device__ NKR_MUL_ATTR FpL<P> mul_add(FpL<P> a, FpL<P> b, FpL<P> c, FpL<P> d)
{
    FpL<P> r;
    mont_mul_add<P>(a.v, b.v, c.v, d.v, r.v);
    reduce_once<TwoP<P>>(r.v);
    return r;
}
template <class P>
__device__ __forceinline__ FpL<P> operator+(const FpL<P> &a, const FpL<P> &b)
{
    FpL<P> r;
    add_words(r.v, a.v, b.v);
    reduce_once<TwoP<P>>(r.v);
    return r;
}
template <class P>
__device__ __forceinline__ FpL<P> operator-(const FpL<P> &a, const FpL<P> &b)
{
    Fp<TwoP<P>> x, y;
#pragma unroll
    for (int j = 0; j < 8; ++j) x.v[j] = a.v[j], y.v[j] = b.v[j];
    x = x - y;
    FpL<P> r;
#pragma unroll
    for (int j = 0; j < 8; ++j) r.v[j] = x.v[j];
    return r;
}
template <class P>
__device__ __forceinline__ FpL<P> neg(const FpL<P> &a)
{
    return FpL<P>::zero() - a;
}
template <class P>
__device__ __forceinline__ FpL<P> dbl(const FpL<P> &a)
{
    return a + a;
}

// ---------------------------------------------------------------------------
// Fq2 = Fq[u] / (u^2 + 1)  (libff alt_bn128_Fq2, non_residue = -1)
// ---------------------------------------------------------------------------
struct alignas(32) Fq2 {
    Fq c0, c1;
    __device__ __forceinline__ static Fq2 zero() { return {Fq::zero(), Fq::zero()}; }
    __device__ __forceinline__ static Fq2 one() { return {Fq::one(), Fq::zero()}; }
    __device__ __forceinline__ bool is_zero() const { return c0.is_zero() && c1.is_zero(); }
    __device__ __forceinline__ bool operator==(const Fq2 &o) const
    {
        return c0 == o.c0 && c1 == o.c1;
    }
    __device__ __forceinline__ bool operator!=(const Fq2 &o) const { return !(*this == o); }
};

__device__ __forceinline__ Fq2 operator+(const Fq2 &a, const Fq2 &b)
{
    return {a.c0 + b.c0, a.c1 + b.c1};
}
__device__ __forceinline__ Fq2 operator-(const Fq2 &a, const Fq2 &b)
{
    return {a.c0 - b.c0, a.c1 - b.c1};
}
__device__ __forceinline__ Fq2 neg(const Fq2 &a) { return {neg(a.c0), neg(a.c1)}; }
__device__ __forceinline__ Fq2 reduced(const Fq2 &a) { return {reduced(a.c0), reduced(a.c1)}; }
__device__ __forceinline__ Fq2 dbl(const Fq2 &a) { return {dbl(a.c0), dbl(a.c1)}; }

// Karatsuba with 3 Montgomery products (one three-product call measured slower:
// more registers and a three times larger body)
__device__ __forceinline__ Fq2 operator*(const Fq2 &a, const Fq2 &b)
{
    const Fq v0 = a.c0 * b.c0;
    const Fq v1 = a.c1 * b.c1;
    const Fq s = (a.c0 + a.c1) * (b.c0 + b.c1);
    return {v0 - v1, s - v0 - v1};
}

// (a0 + a1 u)^2 = (a0 + a1)(a0 - a1) + 2 a0 a1 u
__device__ __forceinline__ Fq2 sqr(const Fq2 &a)
{
    const Fq p = (a.c0 + a.c1) * (a.c0 - a.c1);
    const Fq q = a.c0 * a.c1;
    return {p, q + q};
}

namespace lazy {
// 256 x 256 -> 512-bit schoolbook product t[16] (little-endian words): even and odd
// accumulators as in mont_mul, kept in place.  The chain of row i that starts at
// offset k ends with its carry at offset k + 8, a word no earlier chain has
// reached except by its own carry.
__device__ __forceinline__ void mul_wide(const uint32_t *a, const uint32_t *b, uint32_t *t)
{
    uint32_t e[18], o[18]; // o[k] holds word offset k + 1
#pragma unroll
    for (int j = 0; j < 18; ++j) e[j] = o[j] = 0;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        eo_mad(e + i, e[i + 8], a[0], a[2], a[4], a[6], b[i]);
        eo_mad(o + i, o[i + 8], a[1], a[3], a[5], a[7], b[i]);
        eo_mad(o + i, o[i + 8], a[0], a[2], a[4], a[6], b[i + 1]);
        eo_mad(e + i + 2, e[i + 10], a[1], a[3], a[5], a[7], b[i + 1]);
    }
    // t = e + 2^32 o: words 1..8, the carry, words 9..15
    uint32_t c = 0;
    t[0] = e[0];
    uint32_t hi[8]; // words 9..16; the product has none at 16
    add_words_carry(t + 1, e + 1, o, c);
    add_words_carry(hi, e + 9, o + 8, c);
#pragma unroll
    for (int j = 0; j < 7; ++j) t[9 + j] = hi[j];
}

// Montgomery reduction T R^-1 mod p of a 512-bit T < p R: the low half's reduction and the
// high half, below 2p before the conditional subtraction
__device__ __forceinline__ Fq redc_wide(const uint32_t *t)
{
    Fq r;
    uint32_t lo[8];
    redc_low<FqParams>(t, lo);
    add_words(r.v, lo, t + 8);
    reduce_once<FqParams>(r.v);
    return r;
}

// p^2 for BN254's base field, 16 little-endian words
__device__ __forceinline__ uint32_t p2_word(int k)
{
    constexpr uint32_t w[16] = {0x275d69b1u, 0x3b5458a2u, 0x09eac101u, 0xa602072du,
                                0x6d96cadcu, 0x4a50189cu, 0x7a1242c8u, 0x04689e95u,
                                0x34c6b38du, 0x26edfa5cu, 0x16375606u, 0xb00b8551u,
                                0x0348d21cu, 0x599a6f7cu, 0x763cbf9cu, 0x0925c4b8u};
    return w[k];
}
} // namespace lazy

// Fq2 with the lazily reduced product below: same layout and values as Fq2, its
// arithmetic closed over the type.  It is the compute type of lane quads on G2 (the MSM's
// levels after the first, blinding), whose long dependent chains gain from the shorter
// product; the G2 accumulation takes Fq2M, where this product's live values spill
// (100,001 points 1.94 ms, with Fq2M 1.84).
struct Fq2L : Fq2 {
    Fq2L() = default;
    __device__ __forceinline__ Fq2L(const Fq2 &a) : Fq2(a) {}
    __device__ __forceinline__ static Fq2L zero() { return Fq2::zero(); }
    __device__ __forceinline__ static Fq2L one() { return Fq2::one(); }
};
__device__ __forceinline__ Fq2L operator+(const Fq2L &a, const Fq2L &b)
{
    return static_cast<const Fq2 &>(a) + static_cast<const Fq2 &>(b);
}
__device__ __forceinline__ Fq2L operator-(const Fq2L &a, const Fq2L &b)
{
    return static_cast<const Fq2 &>(a) - static_cast<const Fq2 &>(b);
}
__device__ __forceinline__ Fq2L neg(const Fq2L &a) { return neg(static_cast<const Fq2 &>(a)); }
__device__ __forceinline__ Fq2L dbl(const Fq2L &a) { return dbl(static_cast<const Fq2 &>(a)); }
__device__ __forceinline__ Fq2L sqr(const Fq2L &a) { return sqr(static_cast<const Fq2 &>(a)); }

// Fq2 product with lazy reduction: the Karatsuba products are formed as 512-bit
// integers and combined before reduction, 3 schoolbook products and 2
// Montgomery reductions instead of 3 Montgomery products (320 wide multiply-adds
// instead of 384):
//   c0 = REDC(a0 b0 + p^2 - a1 b1)                          T in [0, 2 p^2)
//   c1 = REDC((a0 + a1)(b0 + b1) - a0 b0 - a1 b1)           T = a0 b1 + a1 b0 in [0, 2 p^2)
// with a0 + a1 and b0 + b1 unreduced (< 2p < 2^255) and 2 p^2 < p R, so each
// reduction lands below 2p and one conditional subtraction makes it canonical:
// the result equals the 3-product form bit for bit.
__device__ NKR_MUL_ATTR_FN Fq2L operator*(Fq2L a, Fq2L b)
{
    uint32_t v0[16], v1[16], t[16], w[16];
    lazy::mul_wide(a.c0.v, b.c0.v, v0);
    lazy::mul_wide(a.c1.v, b.c1.v, v1);
    {
        int64_t c0 = 0, c1 = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int64_t d = int64_t(v0[k]) + lazy::p2_word(k) - int64_t(v1[k]) + c0;
            t[k] = uint32_t(d);
            c0 = d >> 32;
            const int64_t e = int64_t(v0[k]) + int64_t(v1[k]) + c1;
            w[k] = uint32_t(e);
            c1 = e >> 32;
        }
    }
    Fq2 r;
    r.c0 = lazy::redc_wide(t);
    uint32_t sa[8], sb[8];
    {
        uint64_t ca = 0, cb = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint64_t x = uint64_t(a.c0.v[k]) + a.c1.v[k] + ca;
            sa[k] = uint32_t(x);
            ca = x >> 32;
            const uint64_t y = uint64_t(b.c0.v[k]) + b.c1.v[k] + cb;
            sb[k] = uint32_t(y);
            cb = y >> 32;
        }
    }
    lazy::mul_wide(sa, sb, t);
    {
        int64_t c = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int64_t d = int64_t(t[k]) - int64_t(w[k]) + c;
            t[k] = uint32_t(d);
            c = d >> 32;
        }
    }
    r.c1 = lazy::redc_wide(t);
    return r;
}


// Fq2 on coordinates below 2p, the compute type of the G2 accumulation: each coordinate of a
// product is a sum of two products with one reduction (mul_add), 384 wide multiply-adds
// like three separate products, without the additions and conditional subtractions of
// Karatsuba's form and with half its live values
struct Fq2M {
    FqL c0, c1;
    Fq2M() = default;
    __device__ __forceinline__ Fq2M(const FqL &a, const FqL &b) : c0(a), c1(b) {}
    __device__ __forceinline__ Fq2M(const Fq2 &a) : c0(a.c0), c1(a.c1) {}
    __device__ __forceinline__ static Fq2M zero() { return Fq2::zero(); }
    __device__ __forceinline__ static Fq2M one() { return Fq2::one(); }
    __device__ __forceinline__ bool is_zero() const { return c0.is_zero() && c1.is_zero(); }
    __device__ __forceinline__ Fq2 canon() const { return {c0.canon(), c1.canon()}; }
    __device__ __forceinline__ bool operator==(const Fq2M &o) const { return c0 == o.c0 && c1 == o.c1; }
};
__device__ __forceinline__ Fq2M operator+(const Fq2M &a, const Fq2M &b) { return {a.c0 + b.c0, a.c1 + b.c1}; }
__device__ __forceinline__ Fq2M operator-(const Fq2M &a, const Fq2M &b) { return {a.c0 - b.c0, a.c1 - b.c1}; }
__device__ __forceinline__ Fq2M neg(const Fq2M &a) { return {neg(a.c0), neg(a.c1)}; }
__device__ __forceinline__ Fq2M dbl(const Fq2M &a) { return {dbl(a.c0), dbl(a.c1)}; }
__device__ __forceinline__ Fq2M operator*(const Fq2M &a, const Fq2M &b)
{
    const FqL x = mul_add(a.c0, b.c0, neg(a.c1), b.c1);
    return {x, mul_add(a.c0, b.c1, a.c1, b.c0)};
}
__device__ __forceinline__ Fq2M sqr(const Fq2M &a)
{
    const FqL x = (a.c0 + a.c1) * (a.c0 - a.c1);
    return {x, dbl(a.c0 * a.c1)};
}

__device__ inline Fq2 inverse(const Fq2 &a)
{
    const Fq n = sqr(a.c0) + sqr(a.c1);
    const Fq ni = inverse(n);
    return {a.c0 * ni, neg(a.c1) * ni};
}

} // namespace nkr
