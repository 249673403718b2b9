// Pippenger MSM kernels (design notes in msm.cuh).
//
// The curve arithmetic here chains many field products per thread, so the
// product is compiled out of line (one body per kernel) to keep the hot loops
// resident in the instruction cache.
#define NKR_FIELD_MUL_OUTLINE 1
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "msm.cuh"
#include "pairing.cuh" // twist_frobenius: the endomorphism psi of G2
#include "quad.cuh"
#include "scan.cuh"

namespace nkr {

namespace {

// --------------------------------------------------------------------------
// signed digits
// --------------------------------------------------------------------------

// Signed digits of a canonical scalar x in windows of c bits: the digit of window k < W - 1
// is in [-(2^(c-1) - 1), 2^(c-1)], that of the last one nonnegative (fewer than c bits are
// left there).  With h = 2^(c-1) - 1, digit k + h is the plain c-bit digit of
// x + sum_{k < W-1} h 2^(ck), so that no window needs the carry of the one below.  The sum is
// below 2^255.
__device__ __forceinline__ Fr biased_scalar(const Fr &x, int c, int W)
{
    Fr r;
    uint64_t carry = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        // bits 32 j .. 32 j + 31 of the bias: bit i is set when i % c != c - 1 and i < c (W - 1)
        uint32_t bias = 0;
        for (int k = 32 * j / c; k < W - 1 && k * c < 32 * j + 32; ++k) {
            const int lo = k * c - 32 * j;
            const uint64_t h = (uint64_t(1) << (c - 1)) - 1;
            bias |= uint32_t(lo >= 0 ? h << lo : h >> -lo);
        }
        carry += uint64_t(x.v[j]) + bias;
        r.v[j] = uint32_t(carry);
        carry >>= 32;
    }
    return r;
}

// digit of window k of a biased scalar: calls f(has, bucket_in_set, negative)
template <class Fn>
__device__ __forceinline__ void with_digit(const Fr &s, int c, int W, int k, Fn &&f)
{
    const int off = k * c, limb = off >> 5, sh = off & 31;
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        lo = j == limb ? s.v[j] : lo;
        hi = j == limb + 1 ? s.v[j] : hi;
    }
    const int bits = int(__funnelshift_r(lo, hi, sh) & ((1u << c) - 1u));
    const int d = k < W - 1 ? bits - ((1 << (c - 1)) - 1) : bits;
    f(d != 0, uint32_t((d < 0 ? -d : d) - 1), d < 0);
}

// Lanes of this warp whose scalar equals this lane's (all eight words): equal
// scalars have equal digits, so one lane per group updates the bucket counters
// for the whole group.  Matching once per scalar replaces a match per digit
// (repeated scalars are what makes buckets hot in sparse witnesses; distinct
// uniform scalars form groups of one).
__device__ __forceinline__ unsigned equal_scalar_lanes(unsigned mask, const Fr &s)
{
    unsigned peers = mask;
#pragma unroll
    for (int w = 0; w < 8; w += 2)
        peers &= __match_any_sync(mask, uint64_t(s.v[w]) | (uint64_t(s.v[w + 1]) << 32));
    return peers;
}

// One scalar per thread; canon keeps the biased scalars for the scatter.  A zero scalar
// (a class member's is added by the class path) is stored as zero and has no digits.
__global__ void k_digits_count(const Fr *__restrict__ scalars, const uint32_t *__restrict__ gather,
                               const uint32_t *__restrict__ class_of, uint64_t n, int c, int W,
                               bool folded, uint32_t B, Fr *__restrict__ canon,
                               uint32_t *__restrict__ counts)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const bool live = i < n;
    Fr s = Fr::zero();
    if (live) {
        const uint64_t v = gather ? gather[i] : i;
        if (!class_of || class_of[v] == kNoClass) s = from_mont(scalars[v]);
    }
    const bool some = !s.is_zero();
    if (some) s = biased_scalar(s, c, W);
    if (live) canon[i] = s;
    const int lane = threadIdx.x & 31;
    const unsigned act = __ballot_sync(0xffffffffu, some);
    if (!some) return;
    const unsigned peers = equal_scalar_lanes(act, s);
    if (lane != __ffs(peers) - 1) return;
    const uint32_t group = uint32_t(__popc(peers));
    for (int k = 0; k < W; ++k)
        with_digit(s, c, W, k, [&](bool has, uint32_t b, bool) {
            if (has) atomicAdd(&counts[(folded ? 0u : uint32_t(k) * B) + b], group);
        });
}

// Windows [wn blockIdx.y, wn (blockIdx.y + 1)) of one scalar per thread.  A thread's atomics
// return a slot each and follow one another, about 0.6 us apart, so few scalars spread
// their windows over more threads (kScatterThreads).
__global__ void k_scatter(const Fr *__restrict__ canon, uint64_t n, int c, int W, bool folded,
                          uint32_t B, int wn, uint32_t *__restrict__ cursor, uint32_t *__restrict__ entries)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const Fr s = i < n ? canon[i] : Fr::zero();
    const bool some = !s.is_zero();
    const unsigned act = __ballot_sync(0xffffffffu, some);
    if (!some) return;
    const unsigned peers = equal_scalar_lanes(act, s);
    const int leader = __ffs(peers) - 1;
    const uint32_t group = uint32_t(__popc(peers));
    const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
    const int k0 = int(blockIdx.y) * wn;
    for (int k = k0; k < min(k0 + wn, W); ++k)
        with_digit(s, c, W, k, [&](bool has, uint32_t b, bool negd) {
            // the group's lanes agree on every digit, so they take this branch together
            if (has) {
                const uint32_t bucket = (folded ? 0u : uint32_t(k) * B) + b;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(&cursor[bucket], group);
                base = __shfl_sync(peers, base, leader);
                const uint32_t point = folded ? uint32_t(uint64_t(k) * n + i) : uint32_t(i);
                entries[base + rank] = point | (negd ? 0x80000000u : 0u);
            }
        });
}
// threads of a scatter: a few warps per scheduler
constexpr uint64_t kScatterThreads = 148 * 4 * 32 * 4;

// --------------------------------------------------------------------------
// storage vs compute.  Every MSM buffer (bases, partials, buckets, reduction items)
// holds canonical values of Fq or Fq2.  Level 1 computes on values below 2p, in FqL (G1) and
// Fq2M (G2), the levels after it on quads of lanes (quad.cuh) in FqL and Fq2L, the canonical
// Fq2 product with two reductions instead of three.
// --------------------------------------------------------------------------

template <class F>
struct MsmArith;
template <>
struct MsmArith<Fq> {
    using type = FqL;
    using quad = FqL;
};
template <>
struct MsmArith<Fq2> {
    using type = Fq2M;
    using quad = Fq2L;
};
template <class F>
using CF = typename MsmArith<F>::type;
template <class F>
using QF = typename MsmArith<F>::quad;

template <class F>
__device__ constexpr int group_of()
{
    return sizeof(F) == sizeof(Fq) ? 1 : 2;
}

__device__ __forceinline__ Fq msm_out(const FqL &x) { return x.canon(); }
__device__ __forceinline__ Fq2 msm_out(const Fq2 &x) { return x; }
__device__ __forceinline__ Fq2 msm_out(const Fq2M &x) { return x.canon(); }

template <class C>
__device__ __forceinline__ auto stx(const Xyzz<C> &c) -> Xyzz<decltype(msm_out(c.x))>
{
    return {msm_out(c.x), msm_out(c.y), msm_out(c.zz), msm_out(c.zzz)};
}

template <class F>
__device__ __forceinline__ Affine<CF<F>> lda(const Affine<F> &s)
{
    return {CF<F>(s.x), CF<F>(s.y)};
}

// this lane's coordinate of a point in memory, read from L2 (the fix-up levels read
// what other blocks of their own launch wrote)
template <class F>
__device__ __forceinline__ QF<F> quad_ld(const Xyzz<F> *p)
{
    union {
        uint4 w[sizeof(F) / 16];
        F f;
    } u;
    const uint4 *q = reinterpret_cast<const uint4 *>(reinterpret_cast<const F *>(p) + quad_role());
#pragma unroll
    for (unsigned j = 0; j < sizeof(F) / 16; ++j) u.w[j] = __ldcg(q + j);
    return QF<F>(u.f);
}
template <class F>
__device__ __forceinline__ void quad_st(Xyzz<F> *p, const QF<F> &v)
{
    reinterpret_cast<F *>(p)[quad_role()] = msm_out(v);
}

// first index in a[0, n) with a[idx] > x (a nondecreasing)
__device__ __forceinline__ uint32_t upper_bound_u32(const uint32_t *a, uint32_t n, uint32_t x)
{
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] <= x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// --------------------------------------------------------------------------
// bucket accumulation
// --------------------------------------------------------------------------

// Pieces of a bucket at level 1: the bucket's entries [off_b, off_b+1) are cut
// by the fixed segments of K1 entries; a bucket inside one segment is complete,
// otherwise it has one piece per segment it touches.  Piece k of bucket b lives
// in partial slot 2 t (the segment's first run) or 2 t + 1 (its last run).
struct Pieces {
    uint32_t t0, count;
    __device__ __forceinline__ uint64_t slot(const uint32_t off_b, uint32_t k1, uint32_t k) const
    {
        if (k == 0) return off_b == t0 * k1 ? 2ull * t0 : 2ull * t0 + 1;
        return 2ull * (t0 + k);
    }
};

__device__ __forceinline__ Pieces bucket_pieces(const uint32_t *offsets, uint32_t b, uint32_t k1)
{
    const uint32_t lo = offsets[b], hi = offsets[b + 1];
    if (hi == lo) return {0, 0};
    const uint32_t t0 = lo / k1, t1 = (hi - 1) / k1;
    return {t0, t1 - t0 + 1};
}

// Buckets of at most `small` pieces (MsmShape::small_pieces) are summed where they are
// consumed (k_reduce_first); larger ones first go through the fix-up levels (k_fix_up), in
// groups of kFixGroup pieces.  Full buckets (four or more pieces on average) are better
// summed by the many quads of the first reduction level: 2^20 points 3.63 -> 3.41 ms with
// 16 instead of 4.  Where few buckets are large, four pieces at most keep that level
// short: 200,003 sparse scalars 0.60 -> 0.55 ms.
constexpr uint32_t kFixGroup = 4;
constexpr unsigned kFixupBlocks = 148 * 8; // grid cap of the fix-up kernel

// The first-level groups of the large buckets, pushed by level 1, and the arrival
// counters of the levels above: base[0] counts the items {bucket, group}, base + 4
// holds them, and base + 4 + 2 cap has one counter per partial slot (zeroed by level 1).
struct FixList {
    uint32_t *base;
    uint32_t cap;
    __device__ __forceinline__ uint2 *items() const { return reinterpret_cast<uint2 *>(base + 4); }
    __device__ __forceinline__ uint32_t *counters() const { return base + 4 + 2ull * cap; }
    __device__ __forceinline__ void push(uint32_t bucket, uint32_t group) const
    {
        const uint32_t i = atomicAdd(base, 1u);
        if (i < cap) items()[i] = {bucket, group};
    }
};
// a bucket of more than four pieces has at most pieces / kFixGroup + 1 groups and all
// buckets together at most 2 segs pieces
uint32_t fix_cap(uint64_t segs) { return uint32_t(segs + 2); }
size_t fix_bytes(uint64_t segs) { return 16 + 8ull * fix_cap(segs) + 8 * segs; }

// Level-1 accumulators live in shared memory: across the out-of-line product calls of a
// mixed addition their four coordinates would otherwise stay in registers.  Layout:
// structure of arrays, word w of thread i at w * BS + i, so a warp's accesses are
// conflict-free.
//
// G1: FqL coordinates (8 words, below 2p).
template <int BS>
struct SmXyzzFq {
    using point = Affine<FqL>;
    uint32_t *s; // the block's area + threadIdx.x; 32 words per thread
    __device__ __forceinline__ FqL ld(int f) const
    {
        FqL v;
#pragma unroll
        for (int j = 0; j < 8; ++j) v.v[j] = s[(f * 8 + j) * BS];
        return v;
    }
    __device__ __forceinline__ void st(int f, const FqL &v) const
    {
#pragma unroll
        for (int j = 0; j < 8; ++j) s[(f * 8 + j) * BS] = v.v[j];
    }
    __device__ __forceinline__ void set(const Xyzz<FqL> &a) const
    {
        st(0, a.x);
        st(1, a.y);
        st(2, a.zz);
        st(3, a.zzz);
    }
    __device__ __forceinline__ Xyzz<Fq> out() const { return stx(Xyzz<FqL>{ld(0), ld(1), ld(2), ld(3)}); }
    __device__ __forceinline__ static point load(const Affine<Fq> &p) { return lda(p); }
};

// G2: Fq2M coordinates (16 words, each half below 2p).
template <int BS>
struct SmXyzzFq2 {
    using point = Affine<Fq2M>;
    uint32_t *s; // the block's area + threadIdx.x; 64 words per thread
    __device__ __forceinline__ Fq2M ld(int f) const
    {
        Fq2M v;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v.c0.v[j] = s[(f * 16 + j) * BS];
            v.c1.v[j] = s[(f * 16 + 8 + j) * BS];
        }
        return v;
    }
    __device__ __forceinline__ void st(int f, const Fq2M &v) const
    {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            s[(f * 16 + j) * BS] = v.c0.v[j];
            s[(f * 16 + 8 + j) * BS] = v.c1.v[j];
        }
    }
    __device__ __forceinline__ void set(const Xyzz<Fq2M> &a) const
    {
        st(0, a.x);
        st(1, a.y);
        st(2, a.zz);
        st(3, a.zzz);
    }
    __device__ __forceinline__ Xyzz<Fq2> out() const { return stx(Xyzz<Fq2M>{ld(0), ld(1), ld(2), ld(3)}); }
    __device__ __forceinline__ static point load(const Affine<Fq2> &p) { return lda(p); }
};

// a b - c d
__device__ __forceinline__ FqL mul_sub(const FqL &a, const FqL &b, const FqL &c, const FqL &d)
{
    return mul_add(a, b, neg(c), d); // one reduction for both products
}
__device__ __forceinline__ Fq2M mul_sub(const Fq2M &a, const Fq2M &b, const Fq2M &c, const Fq2M &d)
{
    const Fq2M cd = c * d;
    return a * b - cd;
}

// acc + q (madd-2008-s: 8M + 2S) on a shared-memory accumulator, q may be infinity;
// each product comes right before its first use, which keeps few values live.  Bound by the
// multiply pipe, so the squarings (100 wide multiply-adds) and the last coordinate's two
// products with one reduction (192) bring G1's 1,280 down to 1,160: the 2^20 MSM 3.91 ->
// 3.64 ms.  G2 in Fq2M instead of three reduced products per Fq2 product: 100,001 points
// 1.97 -> 1.84 ms, the 2^20 prove 10.0 -> 9.7 ms; in Fq2L (two reductions, 320 instead of
// 384 per product, but more live values and spills) 1.94 ms and 10.0 ms.
template <class Acc, class C>
__device__ __forceinline__ void sm_add_affine(const Acc &a, const Affine<C> &q)
{
    if (q.is_inf()) return;
    const C zz = a.ld(2);
    if (zz.is_zero()) {
        a.set({q.x, q.y, C::one(), C::one()});
        return;
    }
    const C p = q.x * zz - a.ld(0);
    const C r = q.y * a.ld(3) - a.ld(1);
    if (p.is_zero()) {
        a.set(r.is_zero() ? xyzz_from_affine_dbl(q) : Xyzz<C>::inf());
        return;
    }
    const C pp = sqr(p);
    const C ppp = p * pp;
    a.st(3, a.ld(3) * ppp);
    const C qq = a.ld(0) * pp;
    const C ox = sqr(r) - ppp - dbl(qq);
    a.st(0, ox);
    a.st(1, mul_sub(r, qq - ox, a.ld(1), ppp));
    a.st(2, a.ld(2) * pp);
}

// Level 1: thread t sums the fixed segment [t K1, (t+1) K1) of the sorted
// entries, split into runs at bucket boundaries, so every lane of a warp does
// the same number of mixed additions whatever the bucket sizes.  A run that is
// a whole bucket is written to the bucket; the segment's first / last run, when
// its bucket continues outside the segment, goes to partial slot 2t / 2t + 1.  The
// segment of every kFixGroup-th piece of a large bucket puts that group on the fix-up
// list.
template <class Acc, class F>
__device__ __forceinline__ void acc_l1_body(const uint32_t *__restrict__ offsets,
                                            const uint32_t *__restrict__ entries,
                                            const Affine<F> *__restrict__ pts, uint32_t nb,
                                            uint32_t kmax, uint32_t small, Xyzz<F> *__restrict__ partials,
                                            Xyzz<F> *__restrict__ buckets, const FixList &fix, uint32_t t,
                                            const Acc &acc)
{
    using C = decltype(acc.ld(0));
    const uint32_t total = offsets[nb];
    const uint32_t k1 = seg_len(total, kmax, group_of<F>());
    const uint64_t beg64 = uint64_t(t) * k1;
    if (beg64 >= total) return;
    fix.counters()[2ull * t] = 0;
    fix.counters()[2ull * t + 1] = 0;
    const uint32_t beg = uint32_t(beg64);
    const uint32_t end = min(beg + k1, total);
    uint32_t b = upper_bound_u32(offsets, nb + 1, beg) - 1; // offsets[b] <= beg < offsets[b + 1]
    uint32_t bstart = offsets[b], bend = offsets[b + 1];
    bool first = true;
    auto to_partial = [&] {
        partials[2ull * t + (first ? 0 : 1)] = acc.out();
        const uint32_t t0 = bstart / k1, pieces = (bend - 1) / k1 - t0 + 1;
        if (pieces > small && (t - t0) % kFixGroup == 0) fix.push(b, (t - t0) / kFixGroup);
    };
    acc.set(Xyzz<C>::inf());
    // one flat loop with the same trip count in every lane keeps the additions
    // converged; the flush at a bucket boundary is a short divergent branch
    for (uint32_t j = beg; j < end; ++j) {
        if (j == bend) {
            if (bstart >= beg)
                buckets[b] = acc.out(); // the bucket started and ended inside the segment
            else
                to_partial(); // first run, bucket began in an earlier segment
            first = false;
            acc.set(Xyzz<C>::inf());
            // next nonempty bucket: usually adjacent, else search
            ++b;
            int steps = 0;
            while (offsets[b + 1] <= j && steps < 8) {
                ++b;
                ++steps;
            }
            if (offsets[b + 1] <= j) b = upper_bound_u32(offsets, nb + 1, j) - 1;
            bstart = offsets[b];
            bend = offsets[b + 1];
        }
        const uint32_t e = entries[j];
        const Affine<F> base = pts[e & 0x7fffffffu]; // whole: 16-byte vector loads
        typename Acc::point p = Acc::load(base);
        if (e >> 31) p = affine_neg(p);
        sm_add_affine(acc, p);
    }
    if (bstart >= beg && bend <= end)
        buckets[b] = acc.out();
    else
        to_partial();
}

__global__ void __launch_bounds__(128, 4) k_acc_l1_g1(const uint32_t *__restrict__ offsets,
                                                       const uint32_t *__restrict__ entries,
                                                       const Affine<Fq> *__restrict__ pts,
                                                       uint32_t nb, uint32_t kmax, uint32_t small,
                                                       Xyzz<Fq> *__restrict__ partials,
                                                       Xyzz<Fq> *__restrict__ buckets, FixList fix)
{
    __shared__ uint32_t sm[32 * 128];
    acc_l1_body(offsets, entries, pts, nb, kmax, small, partials, buckets, fix,
                blockIdx.x * blockDim.x + threadIdx.x, SmXyzzFq<128>{sm + threadIdx.x});
}

__global__ void __launch_bounds__(128, 3) k_acc_l1_g2(const uint32_t *__restrict__ offsets,
                                                       const uint32_t *__restrict__ entries,
                                                       const Affine<Fq2> *__restrict__ pts,
                                                       uint32_t nb, uint32_t kmax, uint32_t small,
                                                       Xyzz<Fq2> *__restrict__ partials,
                                                       Xyzz<Fq2> *__restrict__ buckets, FixList fix)
{
    __shared__ uint32_t sm[64 * 128];
    acc_l1_body(offsets, entries, pts, nb, kmax, small, partials, buckets, fix,
                blockIdx.x * blockDim.x + threadIdx.x, SmXyzzFq2<128>{sm + threadIdx.x});
}

// Level 1 of several MSMs of one group in one launch (a batch's MSMs, any sizes):
// item i owns blocks [first_block, next item's first_block) of the grid.
template <class F>
struct AccItem {
    const uint32_t *offsets, *entries;
    const Affine<F> *pts;
    Xyzz<F> *partials, *buckets;
    uint32_t *fix_base;
    uint32_t fix_capacity, nb, first_block;
    uint16_t kmax, small;
};
static_assert(sizeof(AccItem<Fq>) <= kMsmAccItemBytes, "work-list item size");

// the work-list item of this block (binary search over the items' first blocks)
template <class F>
__device__ __forceinline__ AccItem<F> acc_list_item(const AccItem<F> *items, int n_items)
{
    int lo = 0, hi = n_items - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (items[mid].first_block <= blockIdx.x)
            lo = mid;
        else
            hi = mid - 1;
    }
    return items[lo];
}

__global__ void __launch_bounds__(128, 4) k_acc_l1_g1_list(const AccItem<Fq> *items, int n_items)
{
    __shared__ uint32_t sm[32 * 128];
    const AccItem<Fq> it = acc_list_item(items, n_items);
    acc_l1_body(it.offsets, it.entries, it.pts, it.nb, it.kmax, it.small, it.partials, it.buckets,
                FixList{it.fix_base, it.fix_capacity},
                (blockIdx.x - it.first_block) * blockDim.x + threadIdx.x, SmXyzzFq<128>{sm + threadIdx.x});
}

__global__ void __launch_bounds__(128, 3) k_acc_l1_g2_list(const AccItem<Fq2> *items, int n_items)
{
    __shared__ uint32_t sm[64 * 128];
    const AccItem<Fq2> it = acc_list_item(items, n_items);
    acc_l1_body(it.offsets, it.entries, it.pts, it.nb, it.kmax, it.small, it.partials, it.buckets,
                FixList{it.fix_base, it.fix_capacity},
                (blockIdx.x - it.first_block) * blockDim.x + threadIdx.x, SmXyzzFq2<128>{sm + threadIdx.x});
}

// The pieces of the large buckets, one launch for all levels: a quad sums a group of
// kFixGroup pieces into the group's first slot and counts itself in at the parent
// group; the quad that arrives last (nobody waits) sums the parent's up to kFixGroup
// children, and so on until the bucket is one piece, which goes to the bucket.  The
// counter of a parent at level l is that of its (l + 1)-th piece: a parent of at least
// two children has more than kFixGroup^l pieces, so these exist and differ per level.
// Every level cost a scan and a launch before (four levels at 2^20 segments), and a
// group took 16 additions by one thread (130 us); a sparse MSM of 200,003 points
// spends 364 us less here.
template <class F>
__global__ void __launch_bounds__(128) k_fix_up(const uint32_t *__restrict__ offsets, uint32_t nb, uint32_t kmax,
                                                 Xyzz<F> *partials, Xyzz<F> *__restrict__ buckets, FixList fix)
{
    using C = QF<F>;
    const uint32_t n = min(*fix.base, fix.cap);
    const uint32_t k1 = seg_len(offsets[nb], kmax, group_of<F>());
    const uint32_t quads = gridDim.x * blockDim.x / 4;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / 4; i < n; i += quads) {
        const uint2 item = fix.items()[i];
        const uint32_t b = item.x;
        uint32_t g = item.y;
        const uint32_t off_b = offsets[b];
        const Pieces pc = bucket_pieces(offsets, b, k1);
        uint64_t stride = 1; // pieces between two inputs of this level
        for (uint32_t level = 1; level <= 16; ++level, stride *= kFixGroup) { // 4^16 pieces at most
            const uint64_t beg = uint64_t(g) * kFixGroup * stride;
            C acc = quad_inf<C>();
            for (uint32_t m = 0; m < kFixGroup; ++m) {
                const uint64_t idx = beg + m * stride;
                if (idx >= pc.count) break;
                acc = quad_add(acc, quad_ld(&partials[pc.slot(off_b, k1, uint32_t(idx))]));
            }
            const uint32_t groups = uint32_t((pc.count + kFixGroup * stride - 1) / (kFixGroup * stride));
            if (groups <= 1) {
                quad_st(&buckets[b], acc);
                break;
            }
            quad_st(&partials[pc.slot(off_b, k1, uint32_t(beg))], acc);
            g /= kFixGroup;
            const uint32_t children = min(kFixGroup, groups - g * kFixGroup);
            if (children > 1) {
                __threadfence();
                __syncwarp(quad_mask());
                uint32_t before = 0;
                if (quad_role() == 0) {
                    const uint64_t piece = uint64_t(g) * kFixGroup * kFixGroup * stride + level;
                    before = atomicAdd(&fix.counters()[pc.slot(off_b, k1, uint32_t(piece))], 1u);
                }
                before = __shfl_sync(quad_mask(), before, 0, 4);
                if (before + 1 != children) break;
                __threadfence();
            }
        }
    }
}

// --------------------------------------------------------------------------
// bucket reduction: sum_b b * S_b per set, then + sum_b S_b
// --------------------------------------------------------------------------

constexpr int kReduceItems = 64; // items (quads) per block of the block levels
constexpr int kReduceLog2 = 6;

// Buckets per quad of the first reduction level (log2): about 2^12 quads per set, two
// thirds of a warp per scheduler, where an addition still runs at its own latency; at
// most 16 buckets, beyond which more quads share the schedulers.  Where a bucket has four
// or more pieces on average, which this level adds up as well, it has enough work for
// 2^14 quads: 2^20 points, 65,536 buckets of 8 pieces, this level 0.78 -> 0.28 ms (and
// 0.47 ms for the fix-up levels instead, had those summed the pieces).
// The environment variable NKR_B200_REDUCE_L2 sets it for tuning experiments.
int first_level_log2(const MsmShape &sh, int bias)
{
    static const int forced = [] {
        const char *e = std::getenv("NKR_B200_REDUCE_L2");
        return e ? std::atoi(e) : -1;
    }();
    const uint32_t m = sh.B;
    int lg = 0;
    while ((uint64_t(1) << (lg + 1)) <= m) ++lg;
    if (forced >= 0) return forced < lg ? forced : lg;
    const int over = lg - (sh.small_pieces > 4 ? 14 : 12);
    int l2 = (over <= 0 ? 0 : over > 4 ? 4 : over) + bias;
    l2 = l2 < 0 ? 0 : l2;
    return l2 < lg ? l2 : lg;
}

// The points that add up to a bucket's sum S_b: none, the whole sum written by level 1 (one
// piece) or by the fix-up levels (more than `small` pieces), or else its few pieces in the
// partial slots.
template <class F>
struct BucketPoints {
    const Xyzz<F> *partials, *whole;
    Pieces pc;
    uint32_t lo, k1, count;
    __device__ __forceinline__ BucketPoints(const uint32_t *__restrict__ offsets, const Xyzz<F> *p,
                                            const Xyzz<F> *buckets, uint32_t b, uint32_t k1_, uint32_t small)
        : partials(p), whole(&buckets[b]), lo(offsets[b]), k1(k1_), count(0)
    {
        const uint32_t hi = offsets[b + 1];
        if (hi == lo) return;
        pc = {lo / k1, (hi - 1) / k1 - lo / k1 + 1};
        count = pc.count;
        if (count > 1 && count <= small)
            whole = nullptr;
        else
            count = 1;
    }
    __device__ __forceinline__ QF<F> get(uint32_t k) const
    {
        return quad_ld(whole ? whole : &partials[pc.slot(lo, k1, k)]);
    }
};

// First reduction level: a quad takes L consecutive buckets and forms
// T = sum_i i S_i and R = sum_i S_i by running sums (2 additions per bucket), emitting
// one (A = T, R) item per L buckets with unit L for the block levels that follow.
// Bucket sums of few pieces are finished here.  All additions go through one place, so
// that quads of a warp in different steps (a piece, a whole bucket, T) add side by side: with
// a place for each, 100,001 points on G2 spent 1.03 instead of 0.21 ms here.
template <class F>
__global__ void __launch_bounds__(128) k_reduce_first(const uint32_t *__restrict__ offsets, uint32_t nb,
                                                       const Xyzz<F> *partials, const Xyzz<F> *buckets,
                                                       uint64_t items, uint32_t L, uint32_t kmax, uint32_t small,
                                                       Xyzz<F> *__restrict__ a_out,
                                                       Xyzz<F> *__restrict__ r_out)
{
    using C = QF<F>;
    const uint64_t t = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / 4;
    if (t * L >= items) return;
    const uint32_t k1 = seg_len(offsets[nb], kmax, group_of<F>());
    const uint64_t base = t * L;
    C run = quad_inf<C>(), tri = quad_inf<C>();
    int i = int(L) - 1;
    BucketPoints<F> pts(offsets, partials, buckets, uint32_t(base + i), k1, small);
    for (uint32_t k = 0;;) {
        const bool point = k < pts.count;
        if (!point && i == 0) break;
        const C sum = quad_add(select(point, run, tri), point ? pts.get(k) : run);
        if (point) {
            run = sum;
            ++k;
        } else {
            tri = sum;
            --i;
            pts = BucketPoints<F>(offsets, partials, buckets, uint32_t(base + i), k1, small);
            k = 0;
        }
    }
    quad_st(&a_out[t], tri);
    quad_st(&r_out[t], run);
}

// A block's points in shared memory, one coordinate per thread: word w of thread j's
// coordinate at w * BS * 4 + j
template <class C, int BS>
struct QuadBuf {
    uint32_t *s;
    static constexpr int words = sizeof(C) / 4;
    __device__ __forceinline__ C ld(int item) const
    {
        union {
            uint32_t w[words];
            C c;
        } u;
        const uint32_t *p = s + item * 4 + quad_role();
#pragma unroll
        for (int j = 0; j < words; ++j) u.w[j] = p[j * BS * 4];
        return u.c;
    }
    __device__ __forceinline__ void st(int item, const C &v) const
    {
        union U {
            uint32_t w[words];
            C c;
            __device__ U() {}
        } u;
        u.c = v;
        uint32_t *p = s + item * 4 + quad_role();
#pragma unroll
        for (int j = 0; j < words; ++j) p[j * BS * 4] = u.w[j];
    }
};

// One level of the weighted sum: items carry (A_c, R_c) with
// S = sum_c (A_c + c U R_c) (unit U = 2^log2_unit).  A block takes BS consecutive
// items c (padding with infinity), one per quad, forms the suffix sums
// Suf_c = sum_{c' >= c} R_c' with a Hillis-Steele scan in shared memory (log2 BS dependent
// additions), then sum_c c R_c = sum_{c >= 1} Suf_c and sum_c A_c by two tree sums on
// disjoint quads, so a level costs about 2 log2(BS) dependent additions.  BS is 64:
// two warps per scheduler, beyond which the products of a step queue for the pipe.
// Output per block: A' = sum A_c + U sum_c c R_c, R' = sum R_c.
template <class F, int BS>
__global__ void __launch_bounds__(BS * 4) k_reduce_block(const Xyzz<F> *__restrict__ a_in,
                                                      const Xyzz<F> *__restrict__ r_in,
                                                      uint32_t m, int log2_unit,
                                                      Xyzz<F> *__restrict__ a_out,
                                                      Xyzz<F> *__restrict__ r_out)
{
    using C = QF<F>;
    extern __shared__ uint32_t sm_words[];
    QuadBuf<C, BS> cur{sm_words}, nxt{sm_words + QuadBuf<C, BS>::words * BS * 4};
    const uint32_t blocks_per_set = (m + BS - 1) / BS;
    const uint32_t set = blockIdx.x / blocks_per_set;
    const uint32_t blk = blockIdx.x % blocks_per_set;
    const int i = threadIdx.x / 4;
    const uint64_t idx = uint64_t(blk) * BS + i;
    const bool live = idx < m;
    const uint64_t g = uint64_t(set) * m + idx;
    C v = live ? quad_ld(&r_in[g]) : quad_inf<C>();
    cur.st(i, v);
    __syncthreads();
    for (int d = 1; d < BS; d <<= 1) {
        if (i + d < BS) v = quad_add(v, cur.ld(i + d));
        nxt.st(i, v);
        __syncthreads();
        const QuadBuf<C, BS> t = cur;
        cur = nxt;
        nxt = t;
    }
    // v = Suf_i.  R' = Suf_0; weighted part = sum_{i >= 1} Suf_i; A part = sum A_i
    nxt.st(i, i >= 1 ? v : quad_inf<C>());
    __syncthreads();
    cur.st(i, live ? quad_ld(&a_in[g]) : quad_inf<C>());
    __syncthreads();
    // the two tree sums side by side on disjoint quads (first s: weighted suffix
    // sums, next s: A items), one addition per quad and step
    for (int s = BS / 2; s > 0; s >>= 1) {
        if (i < s)
            nxt.st(i, quad_add(nxt.ld(i), nxt.ld(i + s)));
        else if (i < 2 * s)
            cur.st(i - s, quad_add(cur.ld(i - s), cur.ld(i)));
        __syncthreads();
    }
    if (i == 0) {
        C w = nxt.ld(0);
        for (int d = 0; d < log2_unit; ++d) w = quad_dbl(w);
        const uint32_t o = set * blocks_per_set + blk;
        quad_st(&a_out[o], quad_add(w, cur.ld(0)));
        quad_st(&r_out[o], v);
    }
}

// XYZZ -> libff Jacobian layout without inversion: with Z = ZZ ZZZ,
// X' = X Z ZZZ and Y' = Y Z^2 ZZ represent the same affine point
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
    const C z = zz * zzz;
    const C t = select(role == 1, z * zz, zzz);
    const C u = v * (z * t); // lane 0: X Z ZZZ, lane 1: Y Z^2 ZZ
    if (role < 3) out[role] = msm_out(role == 2 ? z : u);
}

// The sum of the sets' results, 2^c apart: quad k adds a[k] + r[k], quad 0 runs the Horner
// chain over them (one set: no chain)
constexpr int kFinalSets = 64;
template <class F>
__global__ void __launch_bounds__(4 * kFinalSets) k_finalize(const Xyzz<F> *a, const Xyzz<F> *r, int sets, int c,
                                                              F *out)
{
    using C = QF<F>;
    extern __shared__ uint32_t sm_words[];
    const QuadBuf<C, kFinalSets> sum{sm_words};
    const int i = threadIdx.x / 4;
    if (i < sets) sum.st(i, quad_add(quad_ld(&a[i]), quad_ld(&r[i])));
    __syncthreads();
    if (i > 0) return;
    C acc = sum.ld(sets - 1);
    for (int k = sets - 2; k >= 0; --k) {
        if (!quad_is_inf(acc))
            for (int d = 0; d < c; ++d) acc = quad_dbl(acc);
        acc = quad_add(acc, sum.ld(k));
    }
    quad_store_jacobian<F>(acc, out);
}

// --------------------------------------------------------------------------
// normalisation and window copies
// --------------------------------------------------------------------------

constexpr int kNormChunk = 16;

// libff Jacobian (X, Y, Z): x = X / Z^2, y = Y / Z^3; batch inversion per chunk
template <class F>
__global__ void k_jac_to_affine(const F *__restrict__ jac, Affine<F> *__restrict__ out, uint64_t n)
{
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t beg = t * kNormChunk;
    if (beg >= n) return;
    const int cnt = int(n - beg < uint64_t(kNormChunk) ? n - beg : uint64_t(kNormChunk));
    F pre[kNormChunk];
    F acc = F::one();
    for (int j = 0; j < cnt; ++j) {
        pre[j] = acc;
        const F z = jac[3 * (beg + j) + 2];
        if (!z.is_zero()) acc = acc * z;
    }
    F inv = inverse(acc);
    for (int j = cnt - 1; j >= 0; --j) {
        const uint64_t i = beg + j;
        const F z = jac[3 * i + 2];
        if (z.is_zero()) {
            out[i] = Affine<F>::inf();
            continue;
        }
        const F zi = inv * pre[j];
        inv = inv * z;
        const F zi2 = sqr(zi);
        out[i] = {zi2 * jac[3 * i], (zi2 * zi) * jac[3 * i + 1]}; // coordinates need not be reduced
    }
}

template <class P>
__global__ void k_bitrev_points(const P *__restrict__ in, P *__restrict__ out, int logn)
{
    const uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= (uint64_t(1) << logn)) return;
    const uint32_t r = logn == 0 ? 0u : (__brev(uint32_t(j)) >> (32 - logn));
    out[r] = in[j];
}

template <class F>
int jac_to_affine_t(const void *jac, void *aff, uint64_t n, cudaStream_t st)
{
    if (n == 0) return NKR_B200_OK;
    const uint64_t chunks = (n + kNormChunk - 1) / kNormChunk;
    k_jac_to_affine<F><<<blocks_for(chunks, 64), 64, 0, st>>>(static_cast<const F *>(jac),
                                                               static_cast<Affine<F> *>(aff), n);
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

// Window copies k = 1..W-1 of the points [beg, beg + m): thread i runs the whole
// doubling chain of point beg + i (c (W - 1) doublings, in the MSM's compute
// field) and writes copy k to out[(k - 1) m + i] (XYZZ, storage domain).
template <class F>
__global__ void k_window_chain(const Affine<F> *__restrict__ pts, Xyzz<F> *__restrict__ out,
                               uint64_t beg, uint64_t m, int c, int W)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= m) return;
    using C = CF<F>;
    const Affine<F> s = pts[beg + i];
    if (s.is_inf()) {
        for (int k = 1; k < W; ++k) out[uint64_t(k - 1) * m + i] = Xyzz<F>::inf();
        return;
    }
    Xyzz<C> x = xyzz_from_affine_dbl(lda(s));
    for (int k = 1; k < W; ++k) {
        for (int d = (k == 1 ? 1 : 0); d < c; ++d) x = xyzz_dbl(x);
        out[uint64_t(k - 1) * m + i] = stx(x);
    }
}

// XYZZ copies of k_window_chain -> affine copies k = 1..W-1 in the bases
// (copy k of point beg + i at pts[k n + beg + i]); batch inversion per chunk of
// kNormChunk scratch entries (a chunk may span two copies: the mapping is per entry)
template <class F>
__global__ void k_window_affine(const Xyzz<F> *__restrict__ in, Affine<F> *__restrict__ pts,
                                uint64_t n, uint64_t beg, uint64_t m, uint64_t count)
{
    const uint64_t t = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t first = t * kNormChunk;
    if (first >= count) return;
    const int cnt = int(count - first < uint64_t(kNormChunk) ? count - first : uint64_t(kNormChunk));
    F pre[kNormChunk];
    F acc = F::one();
    for (int j = 0; j < cnt; ++j) {
        pre[j] = acc;
        const Xyzz<F> p = in[first + j];
        if (!p.is_inf()) acc = acc * (p.zz * p.zzz);
    }
    F inv = inverse(acc);
    for (int j = cnt - 1; j >= 0; --j) {
        const uint64_t e = first + j;
        const uint64_t dst = (e / m + 1) * n + beg + e % m;
        const Xyzz<F> p = in[e];
        if (p.is_inf()) {
            pts[dst] = Affine<F>::inf();
            continue;
        }
        const F d = p.zz * p.zzz;
        const F ti = inv * pre[j];
        inv = inv * d;
        pts[dst] = {p.x * (ti * p.zzz), p.y * (ti * p.zz)};
    }
}

// The W - 1 folded window copies 2^(c k) P of every base: per chunk of points one
// launch runs every copy's doublings (so a small key pays one doubling chain and
// one batch inversion, not W - 1 of each) and one launch converts them to affine.
template <class F>
int build_windows_t(MsmBases &b, cudaStream_t st)
{
    const MsmShape &sh = b.shape;
    if (sh.W < 2 || sh.n == 0) return NKR_B200_OK;
    Affine<F> *pts = b.pts.as<Affine<F>>();
    const uint64_t copies = uint64_t(sh.W - 1);
    // scratch of at most ~1 GiB: chunk * copies XYZZ points
    const uint64_t cap = std::max<uint64_t>(1, (uint64_t(1) << 30) / (copies * sizeof(Xyzz<F>)));
    const uint64_t chunk = std::min<uint64_t>(sh.n, cap);
    DevBuf tmp;
    NKR_TRY(tmp.alloc(chunk * copies * sizeof(Xyzz<F>), "window copy scratch"));
    for (uint64_t beg = 0; beg < sh.n; beg += chunk) {
        const uint64_t m = std::min<uint64_t>(chunk, sh.n - beg);
        k_window_chain<F><<<blocks_for(m, 128), 128, 0, st>>>(pts, tmp.as<Xyzz<F>>(), beg, m, sh.c,
                                                              sh.W);
        NKR_CHECK_LAUNCH();
        const uint64_t count = m * copies;
        k_window_affine<F><<<blocks_for((count + kNormChunk - 1) / kNormChunk, 64), 64, 0, st>>>(
            tmp.as<Xyzz<F>>(), pts, sh.n, beg, m, count);
        NKR_CHECK_LAUNCH();
    }
    NKR_CUDA(cudaStreamSynchronize(st));
    return NKR_B200_OK;
}

template <class F>
int launch_level1(uint64_t segs, const uint32_t *offsets, const uint32_t *entries, const Affine<F> *pts, uint32_t nb,
                  uint32_t kmax, uint32_t small, Xyzz<F> *partials, Xyzz<F> *buckets, const DevBuf &fix, cudaStream_t st)
{
    if (segs == 0) return NKR_B200_OK;
    const FixList fl{fix.as<uint32_t>(), fix_cap(segs)};
    NKR_CUDA(cudaMemsetAsync(fl.base, 0, 4, st));
    if constexpr (std::is_same<F, Fq>::value)
        k_acc_l1_g1<<<blocks_for(segs, 128), 128, 0, st>>>(offsets, entries, pts, nb, kmax, small, partials, buckets, fl);
    else
        k_acc_l1_g2<<<blocks_for(segs, 128), 128, 0, st>>>(offsets, entries, pts, nb, kmax, small, partials, buckets, fl);
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

template <class F>
int acc_level1_t(const MsmBases &bs, const MsmSort &s, MsmAcc &a, cudaStream_t st)
{
    const MsmShape &sh = bs.shape;
    // no bucket clearing: a bucket is read only after the kernel that wrote it
    const uint64_t segs = sh.segments_max();
    const uint32_t *offsets = s.offsets.as<uint32_t>();
    if (a.timing) NKR_CUDA(record_timing(a.ev_acc[0], st));
    NKR_TRY(launch_level1<F>(segs, offsets, s.entries.as<uint32_t>(), bs.pts.as<Affine<F>>(), sh.nb,
                             uint32_t(sh.k1), sh.small_pieces, a.partials.as<Xyzz<F>>(), a.buckets.as<Xyzz<F>>(),
                             a.fix, st));
    if (a.timing) NKR_CUDA(record_timing(a.ev_acc[1], st));
    return NKR_B200_OK;
}

// Level 1 of n MSMs of one group in one launch; items_dev is device scratch of n
// work-list items.
template <class F>
int acc_level1_list_t(const MsmAccJob *jobs, int n, void *items_host, void *items_dev, cudaStream_t st)
{
    if (n <= 0) return NKR_B200_OK;
    AccItem<F> *items = static_cast<AccItem<F> *>(items_host);
    uint64_t blocks = 0;
    for (int i = 0; i < n; ++i) {
        const MsmShape &sh = jobs[i].bases->shape;
        AccItem<F> &it = items[i];
        it.offsets = jobs[i].sort->offsets.as<uint32_t>();
        it.entries = jobs[i].sort->entries.as<uint32_t>();
        it.pts = jobs[i].bases->pts.as<Affine<F>>();
        it.partials = jobs[i].acc->partials.as<Xyzz<F>>();
        it.buckets = jobs[i].acc->buckets.as<Xyzz<F>>();
        it.fix_base = jobs[i].acc->fix.as<uint32_t>();
        it.fix_capacity = fix_cap(sh.segments_max());
        it.nb = sh.nb;
        it.kmax = uint16_t(sh.k1);
        it.small = uint16_t(sh.small_pieces);
        if (sh.segments_max()) NKR_CUDA(cudaMemsetAsync(it.fix_base, 0, 4, st));
        it.first_block = uint32_t(blocks);
        blocks += blocks_for(sh.segments_max(), 128);
        NKR_REQUIRE(blocks < (uint64_t(1) << 31), "batched accumulation too large");
    }
    AccItem<F> *d = static_cast<AccItem<F> *>(items_dev);
    NKR_CUDA(cudaMemcpyAsync(d, items, n * sizeof(AccItem<F>), cudaMemcpyHostToDevice, st));
    if constexpr (std::is_same<F, Fq>::value)
        k_acc_l1_g1_list<<<unsigned(blocks), 128, 0, st>>>(d, n);
    else
        k_acc_l1_g2_list<<<unsigned(blocks), 128, 0, st>>>(d, n);
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

// The reduction levels of an MSM whose buckets are final: first level, block
// levels, final combination.
template <class F>
int reduce_run(const MsmBases &bs, const MsmSort &s, MsmAcc &a, void *out_dev, cudaStream_t st)
{
    const MsmShape &sh = bs.shape;
    const uint32_t *offsets = s.offsets.as<uint32_t>();
    const uint32_t sets = sh.folded ? 1u : uint32_t(sh.W);
    NKR_REQUIRE(sets <= uint32_t(kFinalSets), "%u windows exceed the final combination's %d", sets, kFinalSets);
    uint32_t m = sh.B;
    Xyzz<F> *bufs_a[2] = {a.red_a.as<Xyzz<F>>(), a.red_a2.as<Xyzz<F>>()};
    Xyzz<F> *bufs_r[2] = {a.red_r.as<Xyzz<F>>(), a.red_r2.as<Xyzz<F>>()};
    constexpr int BS = kReduceItems;
    const size_t smem = 2 * 4 * BS * sizeof(QF<F>);
    NKR_CUDA(cudaFuncSetAttribute(k_reduce_block<F, BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    // first level: bucket sums (few-piece buckets finished here), L buckets per item
    const int log2_l = first_level_log2(sh, a.first_level_bias);
    const uint32_t L = 1u << log2_l;
    const uint64_t items = uint64_t(sets) * m;
    k_reduce_first<F><<<blocks_for(4 * (items / L), 128), 128, 0, st>>>(
        offsets, sh.nb, a.partials.as<Xyzz<F>>(), a.buckets.as<Xyzz<F>>(), items, L, uint32_t(sh.k1), sh.small_pieces,
        bufs_a[0], bufs_r[0]);
    NKR_CHECK_LAUNCH();
    if (a.timing) NKR_CUDA(record_timing(a.ev_acc[3], st));
    const Xyzz<F> *a_in = bufs_a[0];
    const Xyzz<F> *r_in = bufs_r[0];
    int flip = 1;
    m /= L;
    int log2_unit = log2_l;
    while (m > 1) {
        const uint32_t per_set = (m + BS - 1) / BS;
        k_reduce_block<F, BS><<<sets * per_set, 4 * BS, smem, st>>>(a_in, r_in, m, log2_unit, bufs_a[flip],
                                                                    bufs_r[flip]);
        NKR_CHECK_LAUNCH();
        a_in = bufs_a[flip];
        r_in = bufs_r[flip];
        flip ^= 1;
        m = per_set;
        log2_unit += kReduceLog2;
    }
    // blocks of the sets' quads only (whole warps)
    k_finalize<F><<<1, sets <= 8 ? 32 : 4 * kFinalSets, 4 * kFinalSets * sizeof(QF<F>), st>>>(
        a_in, r_in, int(sets), sh.c, static_cast<F *>(out_dev));
    NKR_CHECK_LAUNCH();
    if (a.timing) NKR_CUDA(record_timing(a.ev_acc[4], st));
    return NKR_B200_OK;
}

// Fix-up levels of a level-1 accumulation with shape sh (segments, buckets, k1) whose
// bucket offsets are `offsets`
template <class F>
int fixup_t(const MsmShape &sh, const uint32_t *offsets, Xyzz<F> *partials, Xyzz<F> *buckets, const DevBuf &fix,
            cudaStream_t st)
{
    const uint64_t segs = sh.segments_max();
    if (segs <= sh.small_pieces) return NKR_B200_OK; // no bucket has more pieces than segments
    const FixList fl{fix.as<uint32_t>(), fix_cap(segs)};
    const unsigned grid = std::min<unsigned>(blocks_for(4ull * fl.cap, 128), kFixupBlocks);
    k_fix_up<F><<<grid, 128, 0, st>>>(offsets, sh.nb, uint32_t(sh.k1), partials, buckets, fl);
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

template <class F>
int acc_tail_t(const MsmBases &bs, const MsmSort &s, MsmAcc &a, void *out_dev, cudaStream_t st)
{
    NKR_TRY(fixup_t<F>(bs.shape, s.offsets.as<uint32_t>(), a.partials.as<Xyzz<F>>(), a.buckets.as<Xyzz<F>>(), a.fix,
                       st));
    if (a.timing) NKR_CUDA(record_timing(a.ev_acc[2], st));
    return reduce_run<F>(bs, s, a, out_dev, st);
}

template <class F>
int acc_run_t(const MsmBases &bs, const MsmSort &s, MsmAcc &a, void *out_dev, cudaStream_t st)
{
    NKR_TRY(acc_level1_t<F>(bs, s, a, st));
    return acc_tail_t<F>(bs, s, a, out_dev, st);
}

template <class F>
int acc_alloc_t(MsmAcc &a, const MsmShape &sh)
{
    const uint32_t sets = sh.folded ? 1u : uint32_t(sh.W);
    // first reduction level output: one item per L buckets
    const uint64_t red = uint64_t(sets) * (sh.B >> first_level_log2(sh, a.first_level_bias)) + 1;
    NKR_TRY(a.partials.alloc(2 * std::max<uint64_t>(sh.segments_max(), 1) * sizeof(Xyzz<F>),
                             "msm partial sums"));
    NKR_TRY(a.buckets.alloc(uint64_t(sh.nb) * sizeof(Xyzz<F>), "msm buckets"));
    NKR_TRY(a.fix.alloc(fix_bytes(sh.segments_max()), "msm fix-up list"));
    NKR_TRY(a.red_a.alloc(red * sizeof(Xyzz<F>), "msm reduction"));
    NKR_TRY(a.red_r.alloc(red * sizeof(Xyzz<F>), "msm reduction"));
    NKR_TRY(a.red_a2.alloc(red * sizeof(Xyzz<F>), "msm reduction"));
    NKR_TRY(a.red_r2.alloc(red * sizeof(Xyzz<F>), "msm reduction"));
    NKR_TRY(a.result.alloc(192, "msm result"));
    return NKR_B200_OK;
}

// --------------------------------------------------------------------------
// repeated scalars: classes of equal witness values (msm.cuh)
// --------------------------------------------------------------------------

__device__ __forceinline__ uint32_t scalar_hash(const Fr &s)
{
    return s.v[0] ^ (s.v[1] * 0x9e3779b9u) ^ (s.v[6] * 0x85ebca6bu) ^ (s.v[7] * 0xc2b2ae35u);
}

constexpr int kDedupProbes = 64; // a value not placed within this many slots stays a singleton

// rep[i]: the representative variable of z_i's value (kNoClass for zero).  The
// table holds variable indices (kNoClass = empty); a thread claims an empty
// slot with atomicCAS or finds an equal value on its probe path.
__global__ void k_dedup_insert(const Fr *__restrict__ z, uint64_t cols, uint32_t *__restrict__ table,
                               uint64_t mask, uint32_t *__restrict__ rep)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= cols) return;
    const Fr s = z[i];
    if (s.is_zero()) {
        rep[i] = kNoClass;
        return;
    }
    uint64_t h = scalar_hash(s) & mask;
    uint32_t r = uint32_t(i);
    for (int probe = 0; probe < kDedupProbes; ++probe) {
        const uint32_t cur = atomicCAS(&table[h], kNoClass, uint32_t(i));
        if (cur == kNoClass) break; // this variable represents its value
        if (z[cur] == s) {
            r = cur;
            break;
        }
        h = (h + 1) & mask;
    }
    rep[i] = r;
}

// csize[r]: members of representative r (warp-aggregated per equal r)
__global__ void k_dedup_count(const uint32_t *__restrict__ rep, uint64_t cols, uint32_t *__restrict__ csize)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t r = i < cols ? rep[i] : kNoClass;
    const unsigned act = __ballot_sync(0xffffffffu, r != kNoClass);
    if (r == kNoClass) return;
    const unsigned peers = __match_any_sync(act, r);
    if (int(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&csize[r], uint32_t(__popc(peers)));
}

// class ids for representatives of at least kClassMin members, first come first
// served up to kClassMax; values[id] = the class's value
__global__ void k_dedup_ids(const Fr *__restrict__ z, const uint32_t *__restrict__ rep,
                            const uint32_t *__restrict__ csize, uint64_t cols, uint32_t *__restrict__ cid,
                            Fr *__restrict__ values, uint32_t *__restrict__ nclass)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= cols) return;
    uint32_t id = kNoClass;
    if (rep[i] == uint32_t(i) && csize[i] >= kClassMin) {
        const uint32_t k = atomicAdd(nclass, 1u);
        if (k < kClassMax) {
            id = k;
            values[k] = z[i];
        }
    }
    cid[i] = id;
}

__global__ void k_dedup_mark(const uint32_t *__restrict__ rep, const uint32_t *__restrict__ cid,
                             uint64_t cols, uint32_t *__restrict__ class_of)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= cols) return;
    const uint32_t r = rep[i];
    class_of[i] = r == kNoClass ? kNoClass : cid[r];
}

// class members of a support: counts per class, then a scatter in class order
// (warp-aggregated per equal class)
__global__ void k_cls_count(const uint32_t *__restrict__ class_of, const uint32_t *__restrict__ gather,
                            uint64_t n, uint32_t *__restrict__ counts)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t c = i < n ? class_of[gather ? gather[i] : i] : kNoClass;
    const unsigned act = __ballot_sync(0xffffffffu, c != kNoClass);
    if (c == kNoClass) return;
    const unsigned peers = __match_any_sync(act, c);
    if (int(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&counts[c], uint32_t(__popc(peers)));
}

__global__ void k_cls_scatter(const uint32_t *__restrict__ class_of, const uint32_t *__restrict__ gather,
                              uint64_t n, uint32_t *__restrict__ cursor, uint32_t *__restrict__ entries)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint32_t c = i < n ? class_of[gather ? gather[i] : i] : kNoClass;
    const unsigned act = __ballot_sync(0xffffffffu, c != kNoClass);
    if (c == kNoClass) return;
    const unsigned peers = __match_any_sync(act, c);
    const int lane = int(threadIdx.x & 31), leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(&cursor[c], uint32_t(__popc(peers)));
    base = __shfl_sync(peers, base, leader);
    entries[base + uint32_t(__popc(peers & ((1u << lane) - 1u)))] = uint32_t(i);
}

// S_c for every class: its pieces (level-1 runs and fix-up sums) added up by a quad and
// normalised with one inversion per class (the quad's lanes run it alike)
template <class F>
__global__ void __launch_bounds__(128) k_cls_finish(const uint32_t *__restrict__ offsets,
                                                     const Xyzz<F> *partials, const Xyzz<F> *buckets, uint32_t kmax,
                                                     uint32_t small, uint32_t nb, Affine<F> *__restrict__ sums)
{
    using C = QF<F>;
    const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) / 4;
    if (c >= nb) return;
    const unsigned role = quad_role();
    const BucketPoints<F> pts(offsets, partials, buckets, c, seg_len(offsets[nb], kmax, group_of<F>()), small);
    C v = quad_inf<C>();
    for (uint32_t k = 0; k < pts.count; ++k) v = quad_add(v, pts.get(k));
    F *out = &sums[c].x;
    if (quad_is_inf(v)) {
        if (role < 2) out[role] = role ? F::one() : F::zero();
        return;
    }
    const C zz = quad_get(v, 2), zzz = quad_get(v, 3);
    const C t = C(inverse(msm_out(zz * zzz)));           // 1 / (ZZ ZZZ)
    const C r = v * (t * select(role == 0, zzz, zz));    // lane 0: X / ZZ, lane 1: Y / ZZZ
    if (role < 2) out[role] = msm_out(r);
}

// acc += add for two libff-Jacobian points (X, Y, Z; Z = 0 is infinity)
template <class F>
__global__ void k_result_add(F *acc, const F *add)
{
    if (threadIdx.x >= 4 || blockIdx.x != 0) return;
    using C = QF<F>;
    const unsigned role = quad_role();
    auto xyzz = [&](const F *p) {
        const C z = C(p[2]), zz = z * z, zzz = zz * z;
        return role < 2 ? C(p[role]) : role == 2 ? zz : zzz;
    };
    quad_store_jacobian<F>(quad_add(xyzz(acc), xyzz(add)), acc);
}

// G2's MSM over its class values uses the twist Frobenius psi(x, y) =
// (conj(x) gx1, conj(y) gy1), which acts on G2 as multiplication by
// lambda = p mod r = 6 u^2 (127 bits): a class value v = k0 + k1 lambda with
// k0 = v mod lambda and k1 = v div lambda (both below 2^128), so the MSM runs over
// the class sums and their images under psi with 128-bit scalars, and its Horner
// chain has half the doublings.
constexpr uint64_t kPsiLambdaLo = 0xf83e9682e87cfd46ull, kPsiLambdaHi = 0x6f4d8248eeb859fbull;
constexpr int kPsiWindows = 13; // 10-bit signed windows over 128-bit scalars (130 bits, no carry out)

__device__ __forceinline__ Fr fr_from_u128(unsigned __int128 x)
{
    Fr r;
#pragma unroll
    for (int i = 0; i < 4; ++i) r.v[i] = uint32_t(x >> (32 * i));
#pragma unroll
    for (int i = 4; i < 8; ++i) r.v[i] = 0;
    return to_mont(r);
}

// values[c] (Montgomery) -> out[c] = k0, out[n + c] = k1 (Montgomery), by binary
// long division of the canonical value by lambda
__global__ void k_cls_split_psi(const Fr *__restrict__ values, uint32_t n, Fr *__restrict__ out)
{
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const Fr v = from_mont(values[c]);
    const unsigned __int128 lam = (unsigned __int128)kPsiLambdaHi << 64 | kPsiLambdaLo;
    unsigned __int128 rem = 0, q = 0;
    for (int i = 253; i >= 0; --i) { // v < r < 2^254; rem < lambda, so 2 rem + 1 < 2^128
        rem = (rem << 1) | ((v.v[i >> 5] >> (i & 31)) & 1u);
        q <<= 1;
        if (rem >= lam) {
            rem -= lam;
            q |= 1;
        }
    }
    out[c] = fr_from_u128(rem);
    out[n + c] = fr_from_u128(q);
}

// sums[n + c] = psi(sums[c]) (infinity stays infinity)
__global__ void k_cls_psi(Affine<Fq2> *sums, uint32_t n)
{
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const Affine<Fq2> a = sums[c];
    sums[n + c] = a.is_inf() ? a : twist_frobenius(a);
}

template <class F>
int class_acc_alloc_t(MsmClassAcc &a, uint64_t n)
{
    a.seg = MsmShape{};
    a.seg.n = n;
    a.seg.c = 1;
    a.seg.W = 1;
    a.seg.folded = true;
    a.seg.B = kClassMax;
    a.seg.nb = kClassMax;
    const uint64_t segs = std::max<uint64_t>(a.seg.segments_max(), 1);
    NKR_TRY(a.partials.alloc(2 * segs * sizeof(Xyzz<F>), "class partial sums"));
    NKR_TRY(a.buckets.alloc(uint64_t(kClassMax) * sizeof(Xyzz<F>), "class sums"));
    NKR_TRY(a.fix.alloc(fix_bytes(segs), "class fix-up list"));
    return NKR_B200_OK;
}

template <class F>
int class_acc_issue_t(const MsmBases &b, const MsmClassSort &cs, MsmClassAcc &a, cudaStream_t st)
{
    const uint64_t segs = a.seg.segments_max();
    const uint32_t *offsets = cs.offsets.as<uint32_t>();
    NKR_TRY(launch_level1<F>(segs, offsets, cs.entries.as<uint32_t>(), b.pts.as<Affine<F>>(), kClassMax,
                             uint32_t(a.seg.k1), a.seg.small_pieces, a.partials.as<Xyzz<F>>(),
                             a.buckets.as<Xyzz<F>>(), a.fix, st));
    NKR_TRY(fixup_t<F>(a.seg, offsets, a.partials.as<Xyzz<F>>(), a.buckets.as<Xyzz<F>>(), a.fix, st));
    k_cls_finish<F><<<blocks_for(4ull * kClassMax, 128), 128, 0, st>>>(
        offsets, a.partials.as<Xyzz<F>>(), a.buckets.as<Xyzz<F>>(), uint32_t(a.seg.k1), a.seg.small_pieces,
        kClassMax, a.small.pts.as<Affine<F>>());
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

} // namespace

double msm_work(uint64_t n, int c)
{
    return double(n) * ((255 + c - 1) / c) * 10.0 + double(uint64_t(1) << (c - 1)) * 2.0 * 32.0;
}

MsmShape msm_shape(uint64_t n, bool folded, int group, int c_override)
{
    MsmShape sh;
    sh.n = n;
    sh.folded = folded;
    int lg = 0;
    while ((uint64_t(1) << lg) < n) ++lg;
    int c;
    (void)group; // G1 and G2 share the shape so MSMs over the same scalars share one sort
    if (c_override > 0) {
        c = c_override;
    } else if (folded) {
        double best = 1e300; // one bucket set
        c = 8;
        for (int cc = 8; cc <= 22; ++cc) {
            const double cost = msm_work(n, cc);
            if (cost < best) {
                best = cost;
                c = cc;
            }
        }
    } else {
        c = lg - 5;
    }
    if (c < 4) c = 4;
    if (c > 22) c = 22;
    sh.c = c;
    sh.W = (255 + c - 1) / c;
    sh.B = 1u << (c - 1);
    sh.nb = folded ? sh.B : sh.B * uint32_t(sh.W);
    sh.small_pieces = sh.entries_max() >= uint64_t(4) * sh.k1 * sh.nb ? 16 : 4;
    return sh;
}

int jacobian_to_affine(int group, const void *jac, void *aff, uint64_t n, cudaStream_t st)
{
    return group == 1 ? jac_to_affine_t<Fq>(jac, aff, n, st) : jac_to_affine_t<Fq2>(jac, aff, n, st);
}

int msm_bases_build(MsmBases &b, int group, const void *jac, bool jac_on_device, uint64_t n,
                    bool folded, int c_override, bool bitrev, cudaStream_t st)
{
    NKR_REQUIRE(group == 1 || group == 2, "group must be 1 (G1) or 2 (G2)");
    b.group = group;
    b.shape = msm_shape(n, folded, group, c_override);
    NKR_REQUIRE(!folded || uint64_t(b.shape.W) * n < (uint64_t(1) << 31),
                "folded MSM of %llu points exceeds the 2^31 entry index space",
                (unsigned long long)n);
    const size_t aff_sz = group == 1 ? sizeof(G1Affine) : sizeof(G2Affine);
    const size_t jac_sz = group == 1 ? 96 : 192;
    const uint64_t copies = folded ? uint64_t(b.shape.W) : 1;
    NKR_TRY(b.pts.alloc(std::max<uint64_t>(n, 1) * copies * aff_sz, "msm bases"));
    if (n == 0) return NKR_B200_OK;
    const void *src = jac;
    DevBuf staging;
    if (!jac_on_device) {
        NKR_TRY(staging.alloc(n * jac_sz, "msm base upload"));
        NKR_CUDA(cudaMemcpyAsync(staging.p, jac, n * jac_sz, cudaMemcpyHostToDevice, st));
        src = staging.p;
    }
    NKR_TRY(jacobian_to_affine(group, src, b.pts.p, n, st));
    if (bitrev) {
        const int lg = log2_exact(n);
        NKR_REQUIRE(lg >= 0 && lg <= 31, "bit-reversed bases need a power-of-two count");
        DevBuf tmp;
        NKR_TRY(tmp.alloc(n * aff_sz, "bitrev base scratch"));
        NKR_CUDA(cudaMemcpyAsync(tmp.p, b.pts.p, n * aff_sz, cudaMemcpyDeviceToDevice, st));
        if (group == 1)
            k_bitrev_points<G1Affine><<<blocks_for(n, 256), 256, 0, st>>>(
                tmp.as<G1Affine>(), b.pts.as<G1Affine>(), lg);
        else
            k_bitrev_points<G2Affine><<<blocks_for(n, 256), 256, 0, st>>>(
                tmp.as<G2Affine>(), b.pts.as<G2Affine>(), lg);
        NKR_CHECK_LAUNCH();
        NKR_CUDA(cudaStreamSynchronize(st));
    }
    if (folded) NKR_TRY(group == 1 ? build_windows_t<Fq>(b, st) : build_windows_t<Fq2>(b, st));
    NKR_CUDA(cudaStreamSynchronize(st));
    return NKR_B200_OK;
}

std::vector<uint32_t> msm_support(int group, const void *jac_host, uint64_t n)
{
    const size_t jac_sz = group == 1 ? 96 : 192;
    const size_t z_off = jac_sz / 3 * 2, z_sz = jac_sz / 3;
    const uint8_t *src = static_cast<const uint8_t *>(jac_host);
    std::vector<uint32_t> idx;
    idx.reserve(n);
    for (uint64_t i = 0; i < n; ++i) {
        const uint8_t *z = src + i * jac_sz + z_off;
        bool zero = true;
        for (size_t k = 0; k < z_sz && zero; k += 8) {
            uint64_t w;
            std::memcpy(&w, z + k, 8);
            zero = w == 0;
        }
        if (!zero) idx.push_back(uint32_t(i));
    }
    if (idx.empty() && n) idx.push_back(0); // an all-infinity query still has one (zero) term
    return idx;
}

int msm_bases_build_support(MsmBases &b, int group, const void *jac_host, uint64_t n,
                            std::vector<uint32_t> idx, bool folded, int c_override, cudaStream_t st)
{
    NKR_REQUIRE(group == 1 || group == 2, "group must be 1 (G1) or 2 (G2)");
    NKR_REQUIRE(n < (uint64_t(1) << 32), "support indices are 32-bit");
    NKR_REQUIRE(idx.size() <= n && (n == 0 || !idx.empty()), "support index list does not fit the bases");
    const size_t jac_sz = group == 1 ? 96 : 192;
    const uint8_t *src = static_cast<const uint8_t *>(jac_host);
    std::vector<uint8_t> packed(std::max<size_t>(idx.size(), 1) * jac_sz);
    for (size_t j = 0; j < idx.size(); ++j) {
        NKR_REQUIRE(idx[j] < n, "support index out of range");
        std::memcpy(packed.data() + j * jac_sz, src + uint64_t(idx[j]) * jac_sz, jac_sz);
    }
    NKR_TRY(msm_bases_build(b, group, packed.data(), false, idx.size(), folded, c_override, false, st));
    b.n_full = n;
    NKR_TRY(b.support.alloc(std::max<size_t>(idx.size(), 1) * 4, "msm support indices"));
    if (!idx.empty())
        NKR_CUDA(cudaMemcpyAsync(b.support.p, idx.data(), idx.size() * 4, cudaMemcpyHostToDevice, st));
    NKR_CUDA(cudaStreamSynchronize(st));
    b.support_host = std::move(idx);
    return NKR_B200_OK;
}

int msm_sort_alloc(MsmSort &s, const MsmShape &sh)
{
    NKR_TRY(s.canon.alloc(std::max<uint64_t>(sh.n, 1) * sizeof(Fr), "msm canonical scalars"));
    NKR_TRY(s.counts.alloc((sh.nb + 1) * 4ull, "msm bucket counts"));
    NKR_TRY(s.offsets.alloc((sh.nb + 1) * 4ull, "msm bucket offsets"));
    NKR_TRY(s.cursor.alloc((sh.nb + 1) * 4ull, "msm scatter cursor"));
    NKR_TRY(s.entries.alloc(std::max<uint64_t>(sh.entries_max(), 1) * 4, "msm entries"));
    NKR_TRY(s.scan_tmp.alloc(scan_scratch_words(sh.nb) * 4, "msm scan scratch"));
    return NKR_B200_OK;
}

int msm_acc_alloc(MsmAcc &a, int group, const MsmShape &sh)
{
    return group == 1 ? acc_alloc_t<Fq>(a, sh) : acc_alloc_t<Fq2>(a, sh);
}

int msm_scratch_alloc(MsmScratch &s, int group, const MsmShape &shape)
{
    NKR_TRY(msm_sort_alloc(s.sort, shape));
    NKR_TRY(msm_acc_alloc(s.acc, group, shape));
    return NKR_B200_OK;
}

int msm_sort_run(const MsmShape &sh, MsmSort &s, const void *scalars_dev, cudaStream_t st,
                 const uint32_t *gather, const uint32_t *class_of)
{
    const uint64_t n = sh.n;
    NKR_CUDA(cudaMemsetAsync(s.counts.p, 0, (sh.nb + 1) * 4, st));
    if (n) {
        k_digits_count<<<blocks_for(n, 256), 256, 0, st>>>(
            static_cast<const Fr *>(scalars_dev), gather, class_of, n, sh.c, sh.W, sh.folded, sh.B,
            s.canon.as<Fr>(), s.counts.as<uint32_t>());
        NKR_CHECK_LAUNCH();
    }
    NKR_TRY(scan_exclusive(LoadU32{s.counts.as<uint32_t>()}, sh.nb, s.offsets.as<uint32_t>(),
                           s.cursor.as<uint32_t>(), s.scan_tmp.as<uint32_t>(), st));
    if (n) {
        uint64_t wn = (n * uint64_t(sh.W) + kScatterThreads - 1) / kScatterThreads; // windows per thread
        wn = std::min<uint64_t>(std::max<uint64_t>(wn, 1), sh.W);
        k_scatter<<<dim3(blocks_for(n, 256), unsigned((sh.W + wn - 1) / wn)), 256, 0, st>>>(
            s.canon.as<Fr>(), n, sh.c, sh.W, sh.folded, sh.B, int(wn), s.cursor.as<uint32_t>(),
            s.entries.as<uint32_t>());
        NKR_CHECK_LAUNCH();
    }
    return NKR_B200_OK;
}

int msm_acc_run(const MsmBases &b, const MsmSort &s, MsmAcc &a, void *out_dev, cudaStream_t st)
{
    return b.group == 1 ? acc_run_t<Fq>(b, s, a, out_dev, st) : acc_run_t<Fq2>(b, s, a, out_dev, st);
}

int msm_acc_level1_list(int group, const MsmAccJob *jobs, int n, void *items_host, void *items_dev,
                        cudaStream_t st)
{
    NKR_REQUIRE(group == 1 || group == 2, "group must be 1 (G1) or 2 (G2)");
    for (int i = 0; i < n; ++i)
        NKR_REQUIRE(jobs[i].bases->group == group, "batched accumulation mixes G1 and G2");
    return group == 1 ? acc_level1_list_t<Fq>(jobs, n, items_host, items_dev, st)
                      : acc_level1_list_t<Fq2>(jobs, n, items_host, items_dev, st);
}

int msm_acc_level1(const MsmBases &b, const MsmSort &s, MsmAcc &a, cudaStream_t st)
{
    return b.group == 1 ? acc_level1_t<Fq>(b, s, a, st) : acc_level1_t<Fq2>(b, s, a, st);
}

int msm_acc_tail(const MsmBases &b, const MsmSort &s, MsmAcc &a, void *out_dev, cudaStream_t st)
{
    return b.group == 1 ? acc_tail_t<Fq>(b, s, a, out_dev, st) : acc_tail_t<Fq2>(b, s, a, out_dev, st);
}

int msm_run(const MsmBases &b, MsmScratch &s, const void *scalars_dev, void *out_dev,
            cudaStream_t st)
{
    NKR_TRY(msm_sort_run(b.shape, s.sort, scalars_dev, st, b.gather()));
    return msm_acc_run(b, s.sort, s.acc, out_dev, st);
}

int msm_dedup_alloc(MsmDedup &d, uint64_t cols)
{
    NKR_REQUIRE(cols < uint64_t(kNoClass), "witness of %llu variables too long for 32-bit indices",
                (unsigned long long)cols);
    d.cols = cols;
    d.slots = 1;
    while (d.slots < 2 * cols) d.slots <<= 1;
    const uint64_t c = std::max<uint64_t>(cols, 1);
    NKR_TRY(d.table.alloc(d.slots * 4, "dedup table"));
    NKR_TRY(d.rep.alloc(c * 4, "dedup representatives"));
    NKR_TRY(d.csize.alloc(c * 4, "dedup class sizes"));
    NKR_TRY(d.cid.alloc(c * 4, "dedup class ids"));
    NKR_TRY(d.class_of.alloc(c * 4, "dedup classes"));
    NKR_TRY(d.values.alloc(uint64_t(kClassMax) * sizeof(Fr), "class values"));
    NKR_TRY(d.nclass.alloc(4, "class count"));
    return NKR_B200_OK;
}

int msm_dedup_run(MsmDedup &d, const void *z, cudaStream_t st)
{
    const uint64_t cols = d.cols;
    NKR_CUDA(cudaMemsetAsync(d.table.p, 0xff, d.table.bytes, st));
    NKR_CUDA(cudaMemsetAsync(d.csize.p, 0, d.csize.bytes, st));
    NKR_CUDA(cudaMemsetAsync(d.values.p, 0, d.values.bytes, st));
    NKR_CUDA(cudaMemsetAsync(d.nclass.p, 0, 4, st));
    if (!cols) return NKR_B200_OK;
    const Fr *zf = static_cast<const Fr *>(z);
    const unsigned g = blocks_for(cols, 256);
    k_dedup_insert<<<g, 256, 0, st>>>(zf, cols, d.table.as<uint32_t>(), d.slots - 1, d.rep.as<uint32_t>());
    NKR_CHECK_LAUNCH();
    k_dedup_count<<<g, 256, 0, st>>>(d.rep.as<uint32_t>(), cols, d.csize.as<uint32_t>());
    NKR_CHECK_LAUNCH();
    k_dedup_ids<<<g, 256, 0, st>>>(zf, d.rep.as<uint32_t>(), d.csize.as<uint32_t>(), cols, d.cid.as<uint32_t>(),
                                   d.values.as<Fr>(), d.nclass.as<uint32_t>());
    NKR_CHECK_LAUNCH();
    k_dedup_mark<<<g, 256, 0, st>>>(d.rep.as<uint32_t>(), d.cid.as<uint32_t>(), cols,
                                    d.class_of.as<uint32_t>());
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

int msm_class_sort_alloc(MsmClassSort &s, uint64_t n)
{
    s.n = n;
    NKR_TRY(s.counts.alloc((kClassMax + 1) * 4ull, "class counts"));
    NKR_TRY(s.offsets.alloc((kClassMax + 1) * 4ull, "class offsets"));
    NKR_TRY(s.cursor.alloc((kClassMax + 1) * 4ull, "class cursor"));
    NKR_TRY(s.entries.alloc(std::max<uint64_t>(n, 1) * 4, "class members"));
    NKR_TRY(s.scan_tmp.alloc(scan_scratch_words(kClassMax) * 4, "class scan scratch"));
    return NKR_B200_OK;
}

int msm_class_sort_run(MsmClassSort &s, const MsmDedup &d, const uint32_t *gather, cudaStream_t st)
{
    NKR_CUDA(cudaMemsetAsync(s.counts.p, 0, (kClassMax + 1) * 4ull, st));
    if (s.n)
        k_cls_count<<<blocks_for(s.n, 256), 256, 0, st>>>(d.class_of.as<uint32_t>(), gather, s.n,
                                                            s.counts.as<uint32_t>());
    NKR_CHECK_LAUNCH();
    NKR_TRY(scan_exclusive(LoadU32{s.counts.as<uint32_t>()}, kClassMax, s.offsets.as<uint32_t>(),
                           s.cursor.as<uint32_t>(), s.scan_tmp.as<uint32_t>(), st));
    if (s.n)
        k_cls_scatter<<<blocks_for(s.n, 256), 256, 0, st>>>(d.class_of.as<uint32_t>(), gather, s.n,
                                                              s.cursor.as<uint32_t>(), s.entries.as<uint32_t>());
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

int msm_class_acc_alloc(MsmClassAcc &a, int group, uint64_t n)
{
    NKR_REQUIRE(group == 1 || group == 2, "group must be 1 (G1) or 2 (G2)");
    NKR_TRY(group == 1 ? class_acc_alloc_t<Fq>(a, n) : class_acc_alloc_t<Fq2>(a, n));
    a.small.group = group;
    // 10-bit windows: 26 of them, so the Horner chain that ends the MSM has 25
    // additions between its ~250 doublings (37 for the cost model's 7-bit windows);
    // G2: the class sums and their psi images with 128-bit scalars, 13 windows
    const uint64_t pts = group == 1 ? kClassMax : 2ull * kClassMax;
    a.small.shape = msm_shape(pts, false, group, 10);
    if (group == 2) {
        a.small.shape.W = kPsiWindows;
        a.small.shape.nb = a.small.shape.B * uint32_t(kPsiWindows);
        NKR_TRY(a.split.alloc(pts * sizeof(Fr), "class value halves"));
    }
    NKR_TRY(a.small.pts.alloc(pts * (group == 1 ? sizeof(G1Affine) : sizeof(G2Affine)), "class sums (affine)"));
    NKR_TRY(msm_scratch_alloc(a.small_s, group, a.small.shape));
    NKR_TRY(a.out.alloc(group == 1 ? 96 : 192, "class MSM result"));
    return NKR_B200_OK;
}

int msm_class_acc_issue(const MsmBases &b, const MsmClassSort &cs, const MsmDedup &d, MsmClassAcc &a,
                        cudaStream_t st)
{
    NKR_REQUIRE(b.group == a.small.group, "class path and bases of different groups");
    NKR_REQUIRE(cs.n == a.seg.n, "class sort and class sums of different supports");
    NKR_TRY(b.group == 1 ? class_acc_issue_t<Fq>(b, cs, a, st) : class_acc_issue_t<Fq2>(b, cs, a, st));
    if (b.group == 1) return msm_run(a.small, a.small_s, d.values.p, a.out.p, st);
    const unsigned g = blocks_for(kClassMax, 128);
    k_cls_psi<<<g, 128, 0, st>>>(a.small.pts.as<Affine<Fq2>>(), kClassMax);
    NKR_CHECK_LAUNCH();
    k_cls_split_psi<<<g, 128, 0, st>>>(d.values.as<Fr>(), kClassMax, a.split.as<Fr>());
    NKR_CHECK_LAUNCH();
    return msm_run(a.small, a.small_s, a.split.p, a.out.p, st);
}

int msm_result_add(int group, void *out_dev, const void *add_dev, cudaStream_t st)
{
    NKR_REQUIRE(group == 1 || group == 2, "group must be 1 (G1) or 2 (G2)");
    if (group == 1)
        k_result_add<Fq><<<1, 32, 0, st>>>(static_cast<Fq *>(out_dev), static_cast<const Fq *>(add_dev));
    else
        k_result_add<Fq2><<<1, 32, 0, st>>>(static_cast<Fq2 *>(out_dev), static_cast<const Fq2 *>(add_dev));
    NKR_CHECK_LAUNCH();
    return NKR_B200_OK;
}

} // namespace nkr
