// Groth16 verification on one B200: the reference's verify
// (protocols/groth16/common/src/protocol.cpp:96-108) for a batch of proofs of
// one verification key, six lanes per proof (pairing_lanes.cuh), and the reduced
// pairing as an operator (libff Curve::reduced_pairing).
//
// The reference checks e(A, B) == e(alpha, beta) e(vk_x, gamma) e(C, delta)
// with three reduced pairings, vk_x = ic[0] + sum_j x_j ic[j + 1].  Here each
// proof takes one Miller loop over the three pairs (A, B), (-vk_x, gamma),
// (-C, delta) and one final exponentiation, and compares with the key's
// e(alpha, beta): the same equation in GT, since the final exponentiation is a
// homomorphism.  gamma and delta are fixed per key, so their Miller-loop lines
// are computed once when the key is prepared; per proof only B's lines are
// computed (homogeneous coordinates, no inversion).  vk_x is a multi-scalar
// multiplication over the key's fixed ic points: the key holds the signed 5-bit
// window multiples d 2^(5w) ic[j + 1] (w < 51, d = 1..16, affine), and 8 or 32 lanes per
// proof sum the looked-up points of its public inputs (k_vk_x) before the pairing kernel
// runs.
#define NKR_FIELD_MUL_OUTLINE 1
#include <cstring>

#include "pairing_lanes.cuh"
#include "prover.cuh"

struct nkr_b200_vk {
    nkr_b200_ctx *ctx = nullptr;
    uint64_t n_ic = 0;
    nkr::DevBuf gt;    // e(alpha, beta): libff alt_bn128_Fq12, 384 B
    nkr::DevBuf ic;    // ic[] as G1 affine (R domain)
    nkr::DevBuf lines; // kAteLines lines of gamma, then of delta
    nkr::DevBuf flags; // int[2]: gamma, delta at infinity
    nkr::DevBuf tab;   // [n_ic - 1][51][16] affine d 2^(5w) ic[j + 1]
    nkr::DevBuf io;    // batch staging (grown on demand)
};

namespace nkr {

namespace {

constexpr size_t kProofBytes = 96 + 192 + 96; // A, B, C in libff layout
constexpr int kIcWin = 51, kIcDig = 16;       // signed 5-bit windows of a public input
// up to this many public inputs a proof's vk_x takes 8 lanes, beyond it a warp: 8 lanes
// need a third of the additions for the final sum, 32 are done sooner
constexpr uint64_t kFewInputs = 64;

// libff Jacobian (X, Y, Z) -> affine; Z = 0 is infinity.  Proofs come from anywhere: their
// coordinates need not be reduced, the arithmetic after this wants them to be.
template <class F>
__device__ __forceinline__ Affine<F> libff_to_affine(const F *p)
{
    if (p[2].is_zero()) return Affine<F>::inf();
    if (p[2] == F::one()) return {reduced(p[0]), reduced(p[1])};
    const F zi = inverse(p[2]);
    const F zi2 = sqr(zi);
    return {zi2 * p[0], (zi2 * zi) * p[1]};
}

// gamma (lane 0) and delta (lane 1): Miller-loop lines; lanes also normalise ic
__global__ void __launch_bounds__(32) k_vk_setup(const Fq2 *gd_jac, const Fq *ic_jac, uint64_t n_ic,
                                                 AteLine *lines, int *flags, G1Affine *ic_aff)
{
    const int lane = threadIdx.x;
    for (uint64_t i = lane; i < n_ic; i += 32) ic_aff[i] = libff_to_affine(ic_jac + 3 * i);
    if (lane < 2) {
        const Affine<Fq2> q = libff_to_affine(gd_jac + 3 * lane);
        flags[lane] = q.is_inf() ? 1 : 0;
        if (!q.is_inf()) ate_lines(q, lines + lane * kAteLines);
    }
}

// Q_{j,w} = 2^(5w) ic[j + 1]: thread j runs the doubling chain (XYZZ scratch)
__global__ void __launch_bounds__(64) k_ic_pow(const G1Affine *ic, uint64_t n_pub, G1Xyzz *pow)
{
    const uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= n_pub) return;
    const G1Affine p = ic[j + 1];
    G1Xyzz q = p.is_inf() ? G1Xyzz::inf() : G1Xyzz{p.x, p.y, Fq::one(), Fq::one()};
    for (int w = 0; w < kIcWin; ++w) {
        pow[j * kIcWin + w] = q;
        if (w + 1 < kIcWin)
            for (int d = 0; d < 5; ++d) q = xyzz_dbl(q);
    }
}

// tab[(j * 51 + w) * 16 + d - 1] = d Q_{j,w} (d = 1..16), affine
__global__ void __launch_bounds__(64) k_ic_entries(const G1Xyzz *pow, uint64_t count, G1Affine *tab)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const G1Xyzz q = pow[i / kIcDig];
    const int d = int(i % kIcDig) + 1;
    G1Xyzz acc = G1Xyzz::inf();
    for (int b = 4; b >= 0; --b) {
        acc = xyzz_dbl(acc);
        if ((d >> b) & 1) acc = xyzz_add(acc, q);
    }
    tab[i] = xyzz_to_affine(acc);
}

__device__ __forceinline__ FqL shfl_down_fq(const FqL &a, int off)
{
    FqL r;
#pragma unroll
    for (int k = 0; k < 8; ++k) r.v[k] = __shfl_down_sync(0xffffffffu, a.v[k], off);
    return r;
}

// vk_x of proof i = ic[0] + sum_j x_ij ic[j + 1] in XYZZ coordinates, L lanes per proof: lane
// l sums the table points of digits l, l + L, ... of all public inputs, 51 signed 5-bit
// digits each, and the lanes' sums are added up; no inversion, the pairing takes the
// point as it is.  With one input per lane four inputs left 28 lanes of a warp idle and
// cost 51 dependent additions; 8 lanes per proof for few inputs keep the final sum short.
// Digits: d_w + 15 are the 5-bit digits of x + sum_w 15 32^w, so they need no carry from
// the windows below (the sum is below 2^255).
template <int L>
__global__ void __launch_bounds__(128) k_vk_x(const G1Affine *ic, const G1Affine *tab, uint64_t n_pub,
                                              const Fr *publics, uint64_t count, G1Xyzz *vk_x)
{
    const uint64_t at = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / L;
    const uint64_t i = at < count ? at : count - 1;
    const int lane = threadIdx.x % L;
    Xyzz<FqL> acc = Xyzz<FqL>::inf();
    uint64_t have = ~uint64_t(0); // public input whose biased scalar is in x
    Fr x = Fr::zero();
    for (uint64_t it = lane; it < n_pub * kIcWin; it += L) {
        const uint64_t j = it / kIcWin;
        const int w = int(it % kIcWin);
        if (j != have) {
            have = j;
            x = from_mont(publics[i * n_pub + j]);
            // sum_w 15 32^w over 51 windows: bits 5w .. 5w + 3
            uint64_t c = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                uint32_t bias = 0;
#pragma unroll
                for (int b = 0; b < 32; ++b)
                    if (32 * k + b < 5 * kIcWin && (32 * k + b) % 5 != 4) bias |= 1u << b;
                c += uint64_t(x.v[k]) + bias;
                x.v[k] = uint32_t(c);
                c >>= 32;
            }
        }
        const int off = 5 * w, limb = off >> 5, sh = off & 31;
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            lo = k == limb ? x.v[k] : lo;
            hi = k == limb + 1 ? x.v[k] : hi;
        }
        const int d = int(__funnelshift_r(lo, hi, sh) & 31u) - 15;
        if (d) {
            const G1Affine e = tab[(j * kIcWin + w) * kIcDig + (d < 0 ? -d : d) - 1];
            const Affine<FqL> p{FqL(e.x), FqL(e.y)};
            acc = xyzz_add_affine(acc, d < 0 ? affine_neg(p) : p);
        }
    }
    for (int off = L / 2; off; off >>= 1)
        acc = xyzz_add(acc, Xyzz<FqL>{shfl_down_fq(acc.x, off), shfl_down_fq(acc.y, off), shfl_down_fq(acc.zz, off),
                                      shfl_down_fq(acc.zzz, off)});
    if (lane == 0 && at < count) {
        acc = xyzz_add_affine(acc, Affine<FqL>{FqL(ic[0].x), FqL(ic[0].y)});
        vk_x[i] = acc.is_inf() ? G1Xyzz::inf()
                               : G1Xyzz{acc.x.canon(), acc.y.canon(), acc.zz.canon(), acc.zzz.canon()};
    }
}

// reduced pairings of count (P, Q) pairs, six lanes each
__global__ void __launch_bounds__(32) k_pairing(const Fq *p_jac, const Fq2 *q_jac, uint64_t count, Fq2 *out)
{
    __shared__ uint4 sm[kPairSmemChunks];
    const PairGroup g(sm, threadIdx.x);
    const uint64_t at = uint64_t(blockIdx.x) * kPairGroups + threadIdx.x / kPairLanes;
    const uint64_t i = at < count ? at : count - 1;
    const Affine<Fq> p = libff_to_affine(p_jac + 3 * i);
    const Affine<Fq2> q = libff_to_affine(q_jac + 3 * i);
    if (g.m == 0) {
        g.st(kSlQx, q.x);
        g.st(kSlQy, q.y);
        g.st(kSlNegPx, {neg(p.x), Fq::zero()});
        g.st(kSlPy, {p.y, Fq::zero()});
        g.st(kSlNegPx1, Fq2::zero());
        g.st(kSlNegPx2, Fq2::zero());
    }
    __syncwarp();
    const PairGroup::Fixed off{{nullptr, nullptr}, {false, false}};
    // a point at infinity: all lines are 1, and so is the pairing
    Fq2 f = g.miller(off, !p.is_inf() && !q.is_inf(), false, Fq::zero());
    f = g.final_power(f);
    if (g.live && at < count) out[6 * i + g.tower_index()] = f;
}

// Six lanes per proof: proofs[i] = A (G1), B (G2), C (G1) in libff layout; vk_x[i] from
// k_vk_x.  The line of (-vk_x, gamma) at vk_x = (X / ZZ, Y / ZZZ) is taken times ZZ ZZZ, a
// factor in Fq that the final exponentiation removes.
__global__ void __launch_bounds__(32) k_verify(const Fq2 *gt, const G1Xyzz *vk_x, const AteLine *lines,
                                               const int *flags, const uint8_t *proofs, uint64_t count,
                                               uint8_t *accept)
{
    __shared__ uint4 sm[kPairSmemChunks];
    const PairGroup g(sm, threadIdx.x);
    const int group = min(int(threadIdx.x) / kPairLanes, kPairGroups - 1);
    const uint64_t at = uint64_t(blockIdx.x) * kPairGroups + group;
    const uint64_t i = at < count ? at : count - 1;
    const uint8_t *pr = proofs + i * kProofBytes;
    const Affine<Fq> a = libff_to_affine(reinterpret_cast<const Fq *>(pr));
    const Affine<Fq2> b = libff_to_affine(reinterpret_cast<const Fq2 *>(pr + 96));
    const Affine<Fq> c = libff_to_affine(reinterpret_cast<const Fq *>(pr + 288));
    const G1Xyzz vk = vk_x[i];
    const bool on1 = !a.is_inf() && !b.is_inf();
    const bool on2 = !vk.is_inf() && !flags[0];
    const bool on3 = !c.is_inf() && !flags[1];
    const Fq none = Fq::zero();
    if (g.m == 0) {
        g.st(kSlQx, b.x);
        g.st(kSlQy, b.y);
        g.st(kSlNegPx, {neg(a.x), none});
        g.st(kSlPy, {a.y, none});
    } else if (g.m == 1) {
        g.st(kSlNegPx1, {neg(vk.x * vk.zzz), none});
        g.st(kSlLine + 5, on2 ? Fq2{neg(vk.y * vk.zz), none} : Fq2::one());
    } else if (g.m == 2) {
        g.st(kSlNegPx2, {neg(c.x), none});
        g.st(kSlLine + 10, on3 ? Fq2{neg(c.y), none} : Fq2::one());
    }
    __syncwarp();
    const PairGroup::Fixed fx{{lines, lines + kAteLines}, {on2, on3}};
    Fq2 f = g.miller(fx, on1, true, vk.zz * vk.zzz);
    f = g.final_power(f);
    const unsigned same = __ballot_sync(0xffffffffu, f == gt[g.tower_index()]);
    if (g.live && g.m == 0 && at < count) accept[i] = ((same >> (group * kPairLanes)) & 63u) == 63u;
}

} // namespace

} // namespace nkr

using namespace nkr;

extern "C" {

int nkr_b200_vk_prepare(nkr_b200_ctx *ctx, const nkr_b200_verification_key *vk, nkr_b200_vk **out)
{
    NKR_REQUIRE(ctx && vk && out, "null argument");
    NKR_REQUIRE(vk->alpha_g1_beta_g2 && vk->gamma_g2 && vk->delta_g2 && vk->ic && vk->n_ic >= 1,
                "verification key: every part is required and ic holds at least one point");
    NKR_CUDA(cudaSetDevice(ctx->device));
    auto key = std::make_unique<nkr_b200_vk>();
    key->ctx = ctx;
    key->n_ic = vk->n_ic;
    cudaStream_t st = ctx->stream;
    DevBuf stage;
    NKR_TRY(stage.alloc(2 * 192 + vk->n_ic * 96, "verification key upload"));
    uint8_t *sp = stage.as<uint8_t>();
    NKR_CUDA(cudaMemcpyAsync(sp, vk->gamma_g2, 192, cudaMemcpyHostToDevice, st));
    NKR_CUDA(cudaMemcpyAsync(sp + 192, vk->delta_g2, 192, cudaMemcpyHostToDevice, st));
    NKR_CUDA(cudaMemcpyAsync(sp + 384, vk->ic, vk->n_ic * 96, cudaMemcpyHostToDevice, st));
    NKR_TRY(key->gt.alloc(kFq12Bytes, "e(alpha, beta)"));
    NKR_CUDA(cudaMemcpyAsync(key->gt.p, vk->alpha_g1_beta_g2, kFq12Bytes, cudaMemcpyHostToDevice, st));
    NKR_TRY(key->ic.alloc(vk->n_ic * sizeof(G1Affine), "ic"));
    NKR_TRY(key->lines.alloc(2 * kAteLines * sizeof(AteLine), "gamma / delta lines"));
    NKR_TRY(key->flags.alloc(2 * sizeof(int), "gamma / delta flags"));
    k_vk_setup<<<1, 32, 0, st>>>(reinterpret_cast<const Fq2 *>(sp), reinterpret_cast<const Fq *>(sp + 384),
                                 vk->n_ic, key->lines.as<AteLine>(), key->flags.as<int>(),
                                 key->ic.as<G1Affine>());
    NKR_CHECK_LAUNCH();
    const uint64_t n_pub = vk->n_ic - 1;
    if (n_pub) {
        const uint64_t entries = n_pub * kIcWin * kIcDig;
        NKR_TRY(key->tab.alloc(entries * sizeof(G1Affine), "ic window tables"));
        DevBuf pow;
        NKR_TRY(pow.alloc(n_pub * kIcWin * sizeof(G1Xyzz), "ic window powers"));
        k_ic_pow<<<blocks_for(n_pub, 64), 64, 0, st>>>(key->ic.as<G1Affine>(), n_pub, pow.as<G1Xyzz>());
        NKR_CHECK_LAUNCH();
        k_ic_entries<<<blocks_for(entries, 64), 64, 0, st>>>(pow.as<G1Xyzz>(), entries,
                                                             key->tab.as<G1Affine>());
        NKR_CHECK_LAUNCH();
        NKR_CUDA(cudaStreamSynchronize(st)); // pow is released on return
    }
    NKR_CUDA(cudaStreamSynchronize(st));
    *out = key.release();
    return NKR_B200_OK;
}

int nkr_b200_verify_batch(nkr_b200_vk *vk, const void *public_inputs, uint64_t n_public,
                          const void *proofs, uint64_t count, uint8_t *accept)
{
    NKR_REQUIRE(vk && accept && (count == 0 || proofs), "null argument");
    NKR_REQUIRE(n_public == 0 || count == 0 || public_inputs, "null public inputs");
    if (count == 0) return NKR_B200_OK;
    // the reference rejects a proof whose public input count does not match ic
    if (n_public + 1 != vk->n_ic) {
        std::memset(accept, 0, count);
        return NKR_B200_OK;
    }
    NKR_CUDA(cudaSetDevice(vk->ctx->device));
    cudaStream_t st = vk->ctx->stream;
    // staging: proofs | public inputs | vk_x (XYZZ) | verdicts
    const uint64_t pb = count * kProofBytes, xb = count * n_public * 32, vb = count * sizeof(G1Xyzz);
    NKR_TRY(vk->io.alloc(pb + xb + vb + count, "verification batch"));
    uint8_t *dp = vk->io.as<uint8_t>();
    G1Xyzz *vkx = reinterpret_cast<G1Xyzz *>(dp + pb + xb);
    uint8_t *acc = dp + pb + xb + vb;
    NKR_CUDA(cudaMemcpyAsync(dp, proofs, pb, cudaMemcpyHostToDevice, st));
    if (xb) NKR_CUDA(cudaMemcpyAsync(dp + pb, public_inputs, xb, cudaMemcpyHostToDevice, st));
    const Fr *pub = reinterpret_cast<const Fr *>(dp + pb);
    if (n_public <= kFewInputs)
        k_vk_x<8><<<blocks_for(count * 8, 128), 128, 0, st>>>(vk->ic.as<G1Affine>(), vk->tab.as<G1Affine>(), n_public,
                                                              pub, count, vkx);
    else
        k_vk_x<32><<<blocks_for(count * 32, 128), 128, 0, st>>>(vk->ic.as<G1Affine>(), vk->tab.as<G1Affine>(),
                                                                n_public, pub, count, vkx);
    NKR_CHECK_LAUNCH();
    k_verify<<<blocks_for(count, kPairGroups), 32, 0, st>>>(vk->gt.as<Fq2>(), vkx, vk->lines.as<AteLine>(),
                                                            vk->flags.as<int>(), dp, count, acc);
    NKR_CHECK_LAUNCH();
    NKR_CUDA(cudaMemcpyAsync(accept, acc, count, cudaMemcpyDeviceToHost, st));
    NKR_CUDA(cudaStreamSynchronize(st));
    return NKR_B200_OK;
}

void nkr_b200_vk_free(nkr_b200_vk *vk)
{
    if (!vk) return;
    cudaSetDevice(vk->ctx->device);
    delete vk;
}

int nkr_b200_reduced_pairing(nkr_b200_ctx *ctx, const void *p_g1, const void *q_g2, uint64_t count,
                             void *out_gt)
{
    NKR_REQUIRE(ctx && (count == 0 || (p_g1 && q_g2 && out_gt)), "null argument");
    if (count == 0) return NKR_B200_OK;
    NKR_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    DevBuf buf;
    NKR_TRY(buf.alloc(count * (96 + 192 + kFq12Bytes), "pairing buffers"));
    uint8_t *b = buf.as<uint8_t>();
    NKR_CUDA(cudaMemcpyAsync(b, p_g1, count * 96, cudaMemcpyHostToDevice, st));
    NKR_CUDA(cudaMemcpyAsync(b + count * 96, q_g2, count * 192, cudaMemcpyHostToDevice, st));
    Fq2 *o = reinterpret_cast<Fq2 *>(b + count * 288);
    k_pairing<<<blocks_for(count, kPairGroups), 32, 0, st>>>(reinterpret_cast<const Fq *>(b),
                                                             reinterpret_cast<const Fq2 *>(b + count * 96), count, o);
    NKR_CHECK_LAUNCH();
    NKR_CUDA(cudaMemcpyAsync(out_gt, o, count * kFq12Bytes, cudaMemcpyDeviceToHost, st));
    NKR_CUDA(cudaStreamSynchronize(st));
    return NKR_B200_OK;
}

} // extern "C"
