// Groth16 blinding (common/src/protocol.cpp:85-94) with caller-given r, s:
//   A = alpha1 + ar + r delta1
//   B = beta2 + bs2 + s delta2
//   C = qz + zk + s A + r B1 - r s delta1
//     = qz + zk + s alpha1 + s ar + r beta1 + r bs1 + r s delta1
//
// Seven scalar multiplications, all of them latency chains for a single GPU
// thread if done by double-and-add (a 256-bit chain on G2 is milliseconds).
// Here:
//  - the five multiples of proving-key constants (r delta1, s alpha1, r beta1,
//    rs delta1 on G1, s delta2 on G2) are fixed-base: prepare tabulates
//    d 2^(8j) P for every 8-bit window j < 32 and digit d < 256 (affine), and one
//    block sums the 32 looked-up points in five levels;
//  - the two multiples of proof points (s ar, r bs1) use the GLV endomorphism of
//    BN254 G1 (Gallant, Lambert and Vanstone, CRYPTO 2001): k = k1 + k2 lambda
//    (mod r) with |k1|, |k2| < 2^127, and k P = k1 P + k2 phi(P) with
//    phi(x, y) = (beta x, y).  A prove through nkr_b200_prove (slot 0) ends by
//    tabulating d 2^(8j) P (j < 16, d < 256) for its own ar and bs1 on a side
//    stream, behind the H MSM (glv_tables_issue); when the raw proof handed to
//    the blinding is that proof, one block per point looks up the 32 digits of
//    k1 and k2 and sums them like the fixed bases.  Any other raw proof takes
//    the chain: the two 127-bit halves run as 4-bit window chains from a 16-entry
//    table built in parallel;
//  - four lanes hold a point and share every addition (quad.cuh): all of this is
//    latency, and one thread per point took 5 to 8 us an addition on G1 and 40 us on G2.
// The kernels return A, B, C as Jacobian points; the host normalises them, as it
// does the raw proof.  Results are group elements, so they equal the
// reference's bit for bit once affine-normalised, whatever the addition order.
#define NKR_FIELD_MUL_OUTLINE 1
#include <algorithm>
#include <cstring>

#include "../host/fr_host.hpp"
#include "field52.cuh" // glv_beta's domain
#include "prover.cuh"
#include "quad.cuh"

namespace nkr {

namespace {

constexpr int kWindows = 32;     // 8-bit windows of a fixed-base scalar
constexpr int kDigits = 255;     // nonzero digits per window
constexpr int kFixedG1 = 3;      // alpha1, beta1, delta1
constexpr size_t kTabG1Bytes = size_t(kFixedG1) * kWindows * kDigits * sizeof(G1Affine);
constexpr size_t kTabG2Bytes = size_t(kWindows) * kDigits * sizeof(G2Affine);

// Host-prepared scalars of one blinding.
struct BlindScalars {
    uint32_t fixed[5][8]; // canonical r, s, r, r s, s for r delta1, s alpha1, r beta1, rs delta1, s delta2
    uint32_t glv[4][4];   // |k1|, |k2| of s (for s ar), then of r (for r bs1)
    uint32_t glv_neg;     // bit c: GLV half c is negative
    uint32_t glv_windows; // 4-bit windows of the longest half
    uint32_t pad[2];
};
static_assert(sizeof(BlindScalars) == 240, "BlindScalars layout");

// blind_io (device) and the slot's pinned staging share this layout
constexpr size_t kIoRaw = 0;       // ar, bs1, zk, qz (G1), bs2 (G2): libff, affine-normalised
constexpr size_t kIoScalars = 576; // BlindScalars
constexpr size_t kIoOut = 832;     // A (G1), B (G2), C (G1): libff Jacobian
constexpr size_t kIoBytes = kIoOut + 384;
constexpr size_t kIoSums = 1280;   // BlindSums (device only)
static_assert(kIoScalars + sizeof(BlindScalars) <= kIoOut && kIoBytes <= kBlindStage && kIoBytes <= kIoSums, "io layout");

// a slot's GLV tables (Xyzz<Fq> entries): the bases ar and bs1, their
// powers Q_j = 2^(8j) P (j < 16), then d Q_j for d = 1..255
constexpr int kGlvWin = 16;
constexpr size_t kGlvPow = 2, kGlvTab = kGlvPow + 2 * kGlvWin;
constexpr size_t kGlvEntries = kGlvTab + 2 * kGlvWin * kDigits;

// pk_const layout: alpha1, beta1, delta1 (G1Affine), beta2, delta2 (G2Affine)
constexpr int kPkAlpha1 = 0, kPkBeta1 = 1, kPkDelta1 = 2, kPkBeta2 = 0, kPkDelta2 = 1;

// ---------------------------------------------------------------------------
// GLV constants of BN254 G1, derived from the curve: beta a primitive cube root
// of unity in Fq and lambda the cube root of unity in Fr with
// (beta x, y) = lambda (x, y); (a1, b1), (a2, b2) the short basis of the lattice
// {(a, b) : a + b lambda = 0 mod r} from the extended Euclidean algorithm on
// (r, lambda) (GLV section 4), b1 < 0 < a1, a2, b2, and a1 b2 - a2 b1 = r;
// g1 = round(b2 2^256 / r), g2 = round(-b1 2^256 / r).
// ---------------------------------------------------------------------------

// beta 2^260 mod p in 52-bit limbs (beta = 0x59e26bcea0d48bacd4f263f1acdb5c4f5763473177fffffe)
__device__ __forceinline__ Fq52 glv_beta()
{
    return {{0x917dda1583b6eull, 0xdc45aa1e7dcf6ull, 0x22e6f2c22a573ull, 0xd1f28e9f64523ull,
             0x1e37a68a14ddull}};
}

__device__ __forceinline__ FqL glv_beta_l() { return FqL(from52(r260_to_r256(glv_beta()))); }

constexpr uint64_t kLambda[4] = {0x8b17ea66b99c90ddull, 0x5bfc41088d8daaa7ull, 0xb3c4d79d41a91758ull, 0};
constexpr uint64_t kGlvA1 = 0x89d3256894d213e3ull; // = b2
constexpr uint64_t kGlvA2[2] = {0x0be4e1541221250bull, 0x6f4d8248eeb859fdull};
constexpr uint64_t kGlvB1Abs[2] = {0x8211bbeb7d4f1128ull, 0x6f4d8248eeb859fcull};
constexpr uint64_t kGlvG1[3] = {0xd91d232ec7e0b3d7ull, 0x2ull, 0};
constexpr uint64_t kGlvG2[3] = {0x7a7bd9d4391eb18eull, 0x4ccef014a773d2cfull, 0x2ull};

using u128 = unsigned __int128;

// out[0, na + nb) = a b
void mul_limbs(const uint64_t *a, int na, const uint64_t *b, int nb, uint64_t *out)
{
    for (int i = 0; i < na + nb; ++i) out[i] = 0;
    for (int i = 0; i < na; ++i) {
        u128 carry = 0;
        for (int j = 0; j < nb; ++j) {
            const u128 t = u128(a[i]) * b[j] + out[i + j] + carry;
            out[i + j] = uint64_t(t);
            carry = t >> 64;
        }
        out[i + nb] = uint64_t(carry);
    }
}

u128 load128(const uint64_t *p) { return u128(p[0]) | (u128(p[1]) << 64); }

int bits128(u128 v)
{
    int n = 0;
    while (v) {
        ++n;
        v >>= 1;
    }
    return n;
}

// k (canonical, < r) -> k1 + k2 lambda with |k1|, |k2| < 2^127.  c_i = floor(k g_i /
// 2^256) is within (-1/8, 1 + 1/8) of the exact quotient k b2 / r (resp. -k b1 / r),
// so |k1| < 1.125 (a1 + a2) < 2^126 and |k2| < 1.125 (|b1| + b2) < 2^126: the
// halves are exact in 128-bit two's complement.  Returns false if the identity
// k = k1 + k2 lambda (mod r) fails (it cannot with these constants; checked
// because the result feeds a proof).
bool glv_split(const uint64_t k[4], uint32_t mag1[4], uint32_t mag2[4], bool &neg1, bool &neg2,
               int &bits)
{
    uint64_t p1[7], p2[7];
    mul_limbs(k, 4, kGlvG1, 3, p1);
    mul_limbs(k, 4, kGlvG2, 3, p2);
    const u128 c1 = load128(p1 + 4), c2 = load128(p2 + 4);
    const u128 k1 = load128(k) - c1 * kGlvA1 - c2 * load128(kGlvA2); // mod 2^128
    const u128 k2 = c1 * load128(kGlvB1Abs) - c2 * kGlvA1;
    neg1 = (k1 >> 127) != 0;
    neg2 = (k2 >> 127) != 0;
    const u128 m1 = neg1 ? u128(0) - k1 : k1, m2 = neg2 ? u128(0) - k2 : k2;
    bits = std::max(bits128(m1), bits128(m2));
    for (int i = 0; i < 4; ++i) {
        mag1[i] = uint32_t(m1 >> (32 * i));
        mag2[i] = uint32_t(m2 >> (32 * i));
    }
    const uint64_t w1[4] = {uint64_t(m1), uint64_t(m1 >> 64), 0, 0};
    const uint64_t w2[4] = {uint64_t(m2), uint64_t(m2 >> 64), 0, 0};
    host::Fr f1 = host::from_canonical(w1), f2 = host::from_canonical(w2);
    if (neg1) f1 = -f1;
    if (neg2) f2 = -f2;
    return f1 + f2 * host::from_canonical(kLambda) == host::from_canonical(k);
}

int blind_scalars(const void *r_mont, const void *s_mont, BlindScalars *o)
{
    host::Fr r, s;
    std::memcpy(r.v, r_mont, 32);
    std::memcpy(s.v, s_mont, 32);
    uint64_t rc[4], sc[4], rsc[4];
    host::to_canonical(r, rc);
    host::to_canonical(s, sc);
    host::to_canonical(r * s, rsc);
    std::memset(o, 0, sizeof(*o));
    const uint64_t *fixed[5] = {rc, sc, rc, rsc, sc};
    for (int t = 0; t < 5; ++t)
        std::memcpy(o->fixed[t], fixed[t], 32);
    bool n[4];
    int b_s = 0, b_r = 0;
    if (!glv_split(sc, o->glv[0], o->glv[1], n[0], n[1], b_s) ||
        !glv_split(rc, o->glv[2], o->glv[3], n[2], n[3], b_r)) {
        set_error("blind: GLV decomposition check failed");
        return NKR_B200_EINVAL;
    }
    for (int c = 0; c < 4; ++c) o->glv_neg |= uint32_t(n[c]) << c;
    o->glv_windows = uint32_t((std::max(b_s, b_r) + 3) / 4);
    return NKR_B200_OK;
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------

template <class F>
struct QuadOf;
template <>
struct QuadOf<Fq> {
    using type = FqL;
};
template <>
struct QuadOf<Fq2> {
    using type = Fq2L;
};
template <class F>
using QF = typename QuadOf<F>::type;

__device__ __forceinline__ Fq canonical(const FqL &x) { return x.canon(); }
__device__ __forceinline__ Fq2 canonical(const Fq2L &x) { return x; }

template <class F>
__device__ __forceinline__ QF<F> quad_ld(const Xyzz<F> *p)
{
    return QF<F>(reinterpret_cast<const F *>(p)[quad_role()]);
}
template <class F>
__device__ __forceinline__ void quad_st(Xyzz<F> *p, const QF<F> &v)
{
    reinterpret_cast<F *>(p)[quad_role()] = canonical(v);
}

// an affine point (infinity is (0, one)) as a quad
template <class F>
__device__ __forceinline__ QF<F> quad_of(const Affine<F> &a)
{
    if (a.is_inf()) return quad_inf<QF<F>>();
    const unsigned role = quad_role();
    return role == 0 ? QF<F>(a.x) : role == 1 ? QF<F>(a.y) : QF<F>::one();
}

// a libff point (X, Y, Z): ZZ = Z^2, ZZZ = Z^3
template <class F>
__device__ __forceinline__ QF<F> quad_of_libff(const F *p)
{
    using C = QF<F>;
    const unsigned role = quad_role();
    const C z = C(p[2]), zz = z * z, zzz = zz * z;
    return role < 2 ? C(p[role]) : role == 2 ? zz : zzz;
}

// Jacobian image of an XYZZ point (ZZ^3 = ZZZ^2): (X ZZ^2, Y ZZZ^2, ZZZ) in libff layout;
// infinity as (0, 1, 0)
template <class F>
__device__ __forceinline__ void quad_store_jacobian(const QF<F> &v, F *out)
{
    using C = QF<F>;
    const unsigned role = quad_role();
    if (quad_is_inf(v)) {
        if (role < 3) out[role] = role == 1 ? F::one() : F::zero();
        return;
    }
    const C zz = quad_get(v, 2), zzz = quad_get(v, 3);
    const C t = select(role == 0, zz, zzz);
    const C u = v * (t * t);
    if (role < 3) out[role] = canonical(role == 2 ? zzz : u);
}

// The sum of the block's 32 quads' points, in five levels; valid in quad 0
template <class F>
__device__ __forceinline__ QF<F> block_sum(QF<F> v, Xyzz<F> *sm)
{
    const int q = threadIdx.x / 4;
    for (int half = 16; half; half >>= 1) {
        if (q >= half && q < 2 * half) quad_st(&sm[q], v);
        __syncthreads();
        if (q < half) v = quad_add(v, quad_ld(&sm[q + half]));
        __syncthreads();
    }
    return v;
}

// this quad's term of k P for the fixed base P tabulated in tab ([32][255] affine): quad j
// looks up the digit of window j
template <class F>
__device__ __forceinline__ QF<F> fixed_base_term(const Affine<F> *tab, const uint32_t *k)
{
    const int j = threadIdx.x / 4;
    const uint32_t d = (k[j >> 2] >> (8 * (j & 3))) & 255u;
    return d ? quad_of(tab[j * kDigits + d - 1]) : quad_inf<QF<F>>();
}

// ---------------------------------------------------------------------------
// prepare: fixed-base tables
// ---------------------------------------------------------------------------

// Q_j = 2^(8j) P for the four fixed bases: block w < 3 takes G1 base w (alpha1,
// beta1, delta1), block 3 takes delta2; one quad runs the doubling chain.
template <class F>
__device__ __forceinline__ void fb_chain(const Affine<F> &p, Xyzz<F> *pow)
{
    QF<F> q = quad_of(p);
    for (int j = 0; j < kWindows; ++j) {
        quad_st(&pow[j], q);
        if (j + 1 < kWindows)
            for (int i = 0; i < 8; ++i) q = quad_dbl(q);
    }
}
__global__ void __launch_bounds__(32) k_fb_powers(const uint8_t *pk_const, Xyzz<Fq> *pow1, Xyzz<Fq2> *pow2)
{
    if (threadIdx.x >= 4) return;
    const int w = blockIdx.x;
    if (w < kFixedG1)
        fb_chain(reinterpret_cast<const G1Affine *>(pk_const)[w], pow1 + w * kWindows);
    else
        fb_chain(reinterpret_cast<const G2Affine *>(pk_const + kFixedG1 * sizeof(G1Affine))[kPkDelta2], pow2);
}

// tab[i] = d Q_{i / 255} with d = i % 255 + 1, affine
template <class F>
__global__ void __launch_bounds__(128) k_fb_entries(const Xyzz<F> *pow, Affine<F> *tab, uint32_t count)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const Xyzz<F> q = pow[i / kDigits];
    const uint32_t d = i % kDigits + 1;
    Xyzz<F> acc = Xyzz<F>::inf();
    for (int b = 7; b >= 0; --b) {
        acc = xyzz_dbl(acc);
        if ((d >> b) & 1) acc = xyzz_add(acc, q);
    }
    tab[i] = xyzz_to_affine(acc);
}

// ---------------------------------------------------------------------------
// prove side: GLV tables of the slot's ar and bs1
// ---------------------------------------------------------------------------

// out: the slot's results (libff Jacobian), ar at 0 and bs1 at 96; one quad per point
// (block) runs the doubling chain
__global__ void __launch_bounds__(32) k_glv_pow(const uint8_t *out, Xyzz<Fq> *t)
{
    if (threadIdx.x >= 4) return;
    const int pt = blockIdx.x;
    FqL q = quad_of_libff(reinterpret_cast<const Fq *>(out + 96 * pt));
    quad_st(&t[pt], q);
    for (int j = 0; j < kGlvWin; ++j) {
        quad_st(&t[kGlvPow + pt * kGlvWin + j], q);
        if (j + 1 < kGlvWin)
            for (int i = 0; i < 8; ++i) q = quad_dbl(q);
    }
}

__global__ void __launch_bounds__(128) k_glv_entries(Xyzz<Fq> *t)
{
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / 4;
    if (i >= 2 * kGlvWin * kDigits) return;
    const FqL q = quad_ld(&t[kGlvPow + i / kDigits]);
    const uint32_t d = i % kDigits + 1;
    FqL acc = q;
    for (int b = 30 - __clz(d); b >= 0; --b) { // bits below the top one
        acc = quad_dbl(acc);
        if ((d >> b) & 1) acc = quad_add(acc, q);
    }
    quad_st(&t[kGlvTab + i], acc);
}

// ---------------------------------------------------------------------------
// the blinding kernels.  Sums: blocks 0-3 the G1 fixed-base sums (r delta1,
// s alpha1, r beta1, rs delta1), block 4 the G2 one (s delta2), blocks 5 and 6 s ar
// and r bs1.  Proof: blocks 0, 1, 2 assemble A, B, C.  One block of 7 warps did all of this
// in 0.44 ms with one thread per point, and the tables of ar and bs1 took 0.61 ms: a prove
// and blinding of a 16-step circuit 1.69 -> 0.99 ms, of matmul 32 2.27 -> 1.84 ms.
// ---------------------------------------------------------------------------

struct BlindSums {
    Xyzz<Fq> g1[7]; // the sums of blocks 0-3, 5 and 6 (index 4 unused)
    Xyzz<Fq2> g2;
};

__global__ void __launch_bounds__(128) k_blind_sums(const G1Affine *g1tab, const G2Affine *g2tab,
                                                    const Xyzz<Fq> *glv, const uint8_t *io, BlindSums *sums)
{
    __shared__ Xyzz<Fq2> sm2[32];
    Xyzz<Fq> *sm1 = reinterpret_cast<Xyzz<Fq> *>(sm2);
    const BlindScalars &sc = *reinterpret_cast<const BlindScalars *>(io + kIoScalars);
    const Fq *raw = reinterpret_cast<const Fq *>(io + kIoRaw);
    const int blk = blockIdx.x, q = threadIdx.x / 4;
    if (blk == 4) {
        const Fq2L v = block_sum<Fq2>(fixed_base_term(g2tab, sc.fixed[4]), sm2);
        if (q == 0) quad_st(&sums->g2, v);
        return;
    }
    FqL v;
    if (blk < 4) {
        const int base = blk == 0 ? kPkDelta1 : blk == 1 ? kPkAlpha1 : blk == 2 ? kPkBeta1 : kPkDelta1;
        v = fixed_base_term(g1tab + size_t(base) * kWindows * kDigits, sc.fixed[blk]);
    } else {
        // point pt (ar with s, bs1 with r); GLV halves c0 = 2 pt (k1), c0 + 1 (k2)
        const int pt = blk - 5, c0 = 2 * pt;
        const unsigned role = quad_role();
        const FqL p = quad_of_libff(raw + 3 * pt); // Z is 0 or 1: affine
        const FqL b = quad_ld(&glv[pt]);
        // is p the base the slot's last prove tabulated (x ZZ = X, y ZZZ = Y)?
        const FqL t = p * quad_get(b, int(role | 2u));
        const bool pinf = quad_is_inf(p), binf = quad_is_inf(b);
        const bool same = quad_flag(t == b, 0) && quad_flag(t == b, 1);
        if (pinf || binf ? pinf && binf : same) {
            // quad h * 16 + j: digit j (8 bits) of half h over 2^(8j) P, or phi of it
            const int h = q >> 4, j = q & 15;
            const uint32_t d = (sc.glv[c0 + h][j >> 2] >> (8 * (j & 3))) & 255u;
            v = quad_inf<FqL>();
            if (d) {
                v = quad_ld(&glv[kGlvTab + (pt * kGlvWin + j) * kDigits + d - 1]);
                if (h && role == 0) v = v * glv_beta_l();
                if (((sc.glv_neg >> (c0 + h)) & 1u) && role == 1) v = neg(v);
            }
        } else {
            // quads 0-15 tabulate d P and, quads 16-31, d phi(P) (d < 16); quads 0 and 16
            // run the halves
            const int d = q & 15, h = q >> 4;
            FqL e = quad_inf<FqL>();
            const FqL base = h && role == 0 ? p * glv_beta_l() : p;
            for (int bit = 3; bit >= 0; --bit) {
                e = quad_dbl(e);
                if ((d >> bit) & 1) e = quad_add(e, base);
            }
            quad_st(&sm1[q], e);
            __syncthreads();
            v = quad_inf<FqL>();
            if (d == 0) {
                const int c = c0 + h;
                const bool ng = (sc.glv_neg >> c) & 1u;
                for (int w = int(sc.glv_windows) - 1; w >= 0; --w) {
                    for (int i = 0; i < 4; ++i) v = quad_dbl(v);
                    const uint32_t dig = (sc.glv[c][w >> 3] >> (4 * (w & 7))) & 15u;
                    if (dig) {
                        FqL e1 = quad_ld(&sm1[16 * h + dig]);
                        if (ng && role == 1) e1 = neg(e1);
                        v = quad_add(v, e1);
                    }
                }
            }
            __syncthreads(); // the table is read before block_sum reuses the memory
        }
    }
    v = block_sum<Fq>(v, sm1);
    if (q == 0) quad_st(&sums->g1[blk], v);
}

__global__ void __launch_bounds__(32) k_blind_proof(const BlindSums *sums, const uint8_t *pk_const, uint8_t *io)
{
    const Fq *raw = reinterpret_cast<const Fq *>(io + kIoRaw);
    const G1Affine *pk1 = reinterpret_cast<const G1Affine *>(pk_const);
    const G2Affine *pk2 = reinterpret_cast<const G2Affine *>(pk_const + kFixedG1 * sizeof(G1Affine));
    __shared__ Xyzz<Fq> sm[8];
    const int q = threadIdx.x / 4;
    if (blockIdx.x == 1) { // B = beta2 + bs2 + s delta2
        if (q > 0) return;
        Fq2L b = quad_add(quad_ld(&sums->g2), quad_of(pk2[kPkBeta2]));
        b = quad_add(b, quad_of_libff(reinterpret_cast<const Fq2 *>(io + kIoRaw + 384)));
        quad_store_jacobian(b, reinterpret_cast<Fq2 *>(io + kIoOut + 96));
        return;
    }
    // A = alpha1 + ar + r delta1, C = (s alpha1 + qz) + (s ar + zk) + (r beta1 + r bs1) + rs delta1:
    // one term per quad, summed in three levels
    FqL v = quad_inf<FqL>();
    if (blockIdx.x == 0) {
        if (q == 0) v = quad_ld(&sums->g1[0]);
        if (q == 1) v = quad_of(pk1[kPkAlpha1]);
        if (q == 2) v = quad_of_libff(raw);
    } else {
        if (q < 3) v = quad_ld(&sums->g1[q + 1]);
        if (q == 3 || q == 4) v = quad_ld(&sums->g1[q + 2]);
        if (q == 5) v = quad_of_libff(raw + 9);
        if (q == 6) v = quad_of_libff(raw + 6);
    }
    for (int half = 4; half; half >>= 1) {
        if (q >= half && q < 2 * half) quad_st(&sm[q], v);
        __syncwarp();
        if (q < half) v = quad_add(v, quad_ld(&sm[q + half]));
        __syncwarp();
    }
    if (q == 0) quad_store_jacobian(v, reinterpret_cast<Fq *>(io + kIoOut + (blockIdx.x == 0 ? 0 : 288)));
}

bool is_one(const host::Fq &z) { return z == host::Fq::one(); }

// The values below p of n coordinates (a raw proof comes from the caller; the kernels take
// coordinates below 2p)
void reduce_coordinates(uint8_t *p, int n)
{
    for (int i = 0; i < n; ++i) {
        host::Fq x;
        std::memcpy(x.v, p + 32 * i, 32);
        if (!host::geq_mod<host::FqMod>(x.v)) continue;
        x = x * host::Fq::one();
        std::memcpy(p + 32 * i, x.v, 32);
    }
}

// Affine-normalise a libff point held as Z = 1, Z = 0 (infinity) or anything else.
void normalize_g1_if_needed(uint8_t *p)
{
    host::Fq z;
    std::memcpy(z.v, p + 64, 32);
    if (!z.is_zero() && !is_one(z))
        host::normalize_g1(p);
    else
        reduce_coordinates(p, 2);
}

void normalize_g2_if_needed(uint8_t *p)
{
    host::Fq z0, z1;
    std::memcpy(z0.v, p + 128, 32);
    std::memcpy(z1.v, p + 160, 32);
    const bool inf = z0.is_zero() && z1.is_zero();
    if (!inf && !(is_one(z0) && z1.is_zero()))
        host::normalize_g2(p);
    else
        reduce_coordinates(p, 4);
}

} // namespace

int blind_tables_build(nkr_b200_key *key, cudaStream_t st)
{
    NKR_TRY(key->blind_io.alloc(kIoSums + sizeof(BlindSums), "blinding io"));
    NKR_TRY(key->blind_tab.alloc(kTabG1Bytes + kTabG2Bytes, "fixed-base blinding tables"));
    DevBuf pow;
    NKR_TRY(pow.alloc(kFixedG1 * kWindows * sizeof(Xyzz<Fq>) + kWindows * sizeof(Xyzz<Fq2>),
                      "fixed-base powers"));
    Xyzz<Fq> *pow1 = pow.as<Xyzz<Fq>>();
    Xyzz<Fq2> *pow2 = reinterpret_cast<Xyzz<Fq2> *>(pow1 + kFixedG1 * kWindows);
    k_fb_powers<<<kFixedG1 + 1, 32, 0, st>>>(key->pk_const.as<uint8_t>(), pow1, pow2);
    NKR_CHECK_LAUNCH();
    const uint32_t n1 = kFixedG1 * kWindows * kDigits, n2 = kWindows * kDigits;
    G1Affine *t1 = key->blind_tab.as<G1Affine>();
    G2Affine *t2 = reinterpret_cast<G2Affine *>(key->blind_tab.as<uint8_t>() + kTabG1Bytes);
    k_fb_entries<Fq><<<blocks_for(n1, 128), 128, 0, st>>>(pow1, t1, n1);
    NKR_CHECK_LAUNCH();
    k_fb_entries<Fq2><<<blocks_for(n2, 128), 128, 0, st>>>(pow2, t2, n2);
    NKR_CHECK_LAUNCH();
    NKR_CUDA(cudaStreamSynchronize(st)); // pow is released on return
    return NKR_B200_OK;
}

size_t glv_tables_bytes() { return kGlvEntries * sizeof(Xyzz<Fq>); }

int glv_tables_issue(ProveSlot *sl, cudaStream_t st)
{
    Xyzz<Fq> *t = sl->glv_tab.as<Xyzz<Fq>>();
    k_glv_pow<<<2, 32, 0, st>>>(sl->out.as<uint8_t>(), t);
    NKR_CHECK_LAUNCH();
    k_glv_entries<<<blocks_for(4 * 2 * kGlvWin * kDigits, 128), 128, 0, st>>>(t);
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

int key_blind(nkr_b200_key *key, const nkr_b200_raw_proof *raw, const void *r, const void *s,
              nkr_b200_proof *res)
{
    NKR_REQUIRE(key && raw && r && s && res, "null argument");
    NKR_CUDA(cudaSetDevice(key->ctx->device));
    ProveSlot *sl = key->slots[0].get();
    cudaStream_t s0 = sl->main();
    uint8_t *host = static_cast<uint8_t *>(sl->pinned_out) + kOutBytes;
    // the staging area is free once slot 0's queued work (an earlier blind) is done
    NKR_CUDA(cudaStreamSynchronize(s0));
    std::memcpy(host + kIoRaw + 0, raw->ar, 96);
    std::memcpy(host + kIoRaw + 96, raw->bs1, 96);
    std::memcpy(host + kIoRaw + 192, raw->zk, 96);
    std::memcpy(host + kIoRaw + 288, raw->qz, 96);
    std::memcpy(host + kIoRaw + 384, raw->bs2, 192);
    for (int i = 0; i < 4; ++i) normalize_g1_if_needed(host + kIoRaw + 96 * i);
    normalize_g2_if_needed(host + kIoRaw + 384);
    NKR_TRY(blind_scalars(r, s, reinterpret_cast<BlindScalars *>(host + kIoScalars)));
    uint8_t *io = key->blind_io.as<uint8_t>();
    NKR_CUDA(cudaMemcpyAsync(io, host, kIoScalars + sizeof(BlindScalars), cudaMemcpyHostToDevice, s0));
    const G1Affine *t1 = key->blind_tab.as<G1Affine>();
    const G2Affine *t2 = reinterpret_cast<const G2Affine *>(key->blind_tab.as<uint8_t>() + kTabG1Bytes);
    BlindSums *sums = reinterpret_cast<BlindSums *>(io + kIoSums);
    k_blind_sums<<<7, 128, 0, s0>>>(t1, t2, sl->glv_tab.as<Xyzz<Fq>>(), io, sums);
    NKR_CHECK_LAUNCH();
    k_blind_proof<<<3, 32, 0, s0>>>(sums, key->pk_const.as<uint8_t>(), io);
    NKR_CHECK_LAUNCH();
    NKR_CUDA(cudaMemcpyAsync(host + kIoOut, io + kIoOut, 384, cudaMemcpyDeviceToHost, s0));
    NKR_CUDA(cudaStreamSynchronize(s0));
    uint8_t *o = host + kIoOut;
    host::normalize_g1(o);
    host::normalize_g2(o + 96);
    host::normalize_g1(o + 288);
    std::memcpy(res->a, o, 96);
    std::memcpy(res->b, o + 96, 192);
    std::memcpy(res->c, o + 288, 96);
    return NKR_B200_OK;
}

} // namespace nkr
