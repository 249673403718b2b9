"""Inputs that are not reduced: a caller's 256-bit words stand for their value modulo r or
p.  Scalars, base and proof coordinates, public inputs, matrix values and vectors that an
operation begins by multiplying give the results of their reduced forms, up to the largest
multiple of the modulus that fits 256 bits."""
import numpy as np
import pytest
import torch

import nkr_b200 as nk
import oracle as O

pytestmark = pytest.mark.gpu


def _plus(a, mod, times=None):
    """Each element plus `times` multiples of mod (the most that fit where None)."""
    a = np.ascontiguousarray(a, np.uint64)
    out = []
    for row in a.reshape(-1, 4):
        v = O.limbs_to_int(row)
        out.append(O.int_to_limbs(v + mod * (((1 << 256) - 1 - v) // mod if times is None else times)))
    return np.stack(out).reshape(a.shape)


@pytest.mark.parametrize("times", [1, 4, None])
@pytest.mark.parametrize("group", [1, 2])
def test_msm(ctx, orc, group, times):
    rng = np.random.default_rng(61)
    n = 70
    gen = orc.g1_generator() if group == 1 else orc.g2_generator()
    jac = O.affine_to_jac(group, np.stack([orc.mul_affine(group, gen, k) for k in O.random_fr(n, rng)]))
    sc = O.random_fr(n, rng)
    sc[5] = 0
    want = ctx.msm(group, jac, sc)
    raw = _plus(sc, O.R, times)
    b = nk.MsmBases(ctx, group, jac)
    assert np.array_equal(ctx.msm(group, jac, raw), want)
    assert np.array_equal(b.run(raw)[0], want)
    b.free()
    coords = 2 if group == 1 else 4
    jac2 = jac.reshape(n, -1).copy()
    # sums of two coordinates of Fq2 stay within 256 bits for one multiple
    jac2[:, :4 * coords] = _plus(jac2[:, :4 * coords], O.P, times if group == 1 else 1)
    assert np.array_equal(ctx.msm(group, jac2, raw), want)


@pytest.mark.parametrize("times", [1, 4, None])
def test_coset_transform_scale_and_quotient(ctx, times):
    rng = np.random.default_rng(62)
    for n in (8, 1 << 10):
        x = O.random_fr(n, rng)
        raw = _plus(x, O.R, times)
        for op in (2, 4):
            assert np.array_equal(ctx.ntt(op, raw), ctx.ntt(op, x)), (n, op)
        d = torch.from_numpy(raw.view(np.int64)).cuda()
        o = torch.empty_like(d)
        nk.ntt_noalloc(0, 2, d.data_ptr(), o.data_ptr(), n)
        torch.cuda.synchronize()
        assert np.array_equal(o.cpu().numpy().view(np.uint64), ctx.ntt(2, x)), n


@pytest.mark.parametrize("times", [1, 4, None])
def test_products_and_spmv(ctx, times):
    rng = np.random.default_rng(63)
    for field, mod in ((0, O.R), (1, O.P)):
        a, b = (np.stack([O.int_to_limbs(O.limbs_to_int(v) % mod) for v in O.random_fr(200, rng)]) for _ in range(2))
        want = ctx.field_op(field, 0, a, b)
        assert np.array_equal(ctx.field_op(field, 0, _plus(a, mod, times), b), want)
        assert np.array_equal(ctx.field_op(field, 0, a, _plus(b, mod, times)), want)
        for op in (5, 6):
            assert np.array_equal(ctx.field_op(field, op, _plus(a, mod, times)), ctx.field_op(field, op, a))
    n = 50
    z, vals = O.random_fr(n, rng), O.random_fr(n, rng)
    ptr, col = np.arange(n + 1), rng.permutation(n)
    want = ctx.spmv(n, n, ptr, col, vals, z)
    assert np.array_equal(ctx.spmv(n, n, ptr, col, _plus(vals, O.R, times), z), want)
    assert np.array_equal(ctx.spmv(n, n, ptr, col, vals, _plus(z, O.R, times)), want)


@pytest.mark.parametrize("times", [1, 4, None])
def test_pairing_and_verification(ctx, times):
    rng = np.random.default_rng(64)
    r1 = nk.generate("matmul", 2, 0, seed=9)
    pk, vkp = nk.setup(ctx, r1, O.random_fr(5, rng))
    be = nk.Backend(ctx)
    be.prepare(r1, pk)
    raw = be.prove(r1.witness)
    r, s = O.random_fr(2, rng)
    good = be.blind(raw, r, s)
    proof = np.frombuffer(bytes(good), np.uint64).copy()
    bad = proof.copy()
    bad[36:48], bad[0:12] = proof[0:12], proof[36:48]
    proofs = np.stack([proof, proof, proof, bad])
    proofs[0, 0:8] = _plus(proofs[0, 0:8], O.P, times)      # A
    proofs[1, 36:44] = _plus(proofs[1, 36:44], O.P, times)  # C
    proofs[2, 12:28] = _plus(proofs[2, 12:28], O.P, times)  # B
    proofs[3, 0:8] = _plus(proofs[3, 0:8], O.P, times)
    pub = np.ascontiguousarray(r1.witness[1:1 + r1.public_inputs])
    publics = np.stack([pub, pub, _plus(pub, O.R, times), pub])
    vk = nk.VerifyingKey(ctx, vkp["alpha_g1_beta_g2"], vkp["gamma_g2"], vkp["delta_g2"], vkp["ic"])
    assert vk.verify_batch(publics, proofs).tolist() == [True, True, True, False]
    vk.free()
    p, q = proof[0:12].copy(), proof[12:36].copy()
    want = nk.reduced_pairing(ctx, p[None], q[None])
    p[:8], q[:16] = _plus(p[:8], O.P, times), _plus(q[:16], O.P, times)
    assert np.array_equal(nk.reduced_pairing(ctx, p[None], q[None]), want)
    be.free()


@pytest.mark.parametrize("times", [1, 4, None])
def test_blinding(ctx, times):
    rng = np.random.default_rng(65)
    r1 = nk.generate("matmul", 2, 0, seed=9)
    pk, _ = nk.setup(ctx, r1, O.random_fr(5, rng))
    be = nk.Backend(ctx)
    be.prepare(r1, pk)
    raw = be.prove(r1.witness)
    r, s = O.random_fr(2, rng)
    want = bytes(be.blind(raw, r, s))
    again = type(raw).from_buffer_copy(bytes(raw))
    words = np.frombuffer(again, np.uint64)
    for i in range(4):
        words[12 * i:12 * i + 8] = _plus(words[12 * i:12 * i + 8], O.P, times)
    words[48:64] = _plus(words[48:64], O.P, times)
    assert bytes(be.blind(again, r, s)) == want
    be.free()
