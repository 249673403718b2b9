"""The class path of repeated witness values (circuits of more than 2^16 variables):
variables of equal value form a class whose bases are summed once, and a small MSM over the
class values adds v_c S_c.  The witness MSMs of a key whose toxic waste is known are
(sum_i w_i k_i) G with the k_i from the oracle's setup, so every point has a value computed
without an MSM.  Single proves, batches over several slots of a key and the server."""
import numpy as np
import pytest

import nkr_b200 as nk
import oracle as O

pytestmark = pytest.mark.gpu

RINV = pow(1 << 256, -1, O.R)


def _ints(a):
    b = np.ascontiguousarray(a, np.uint64).tobytes()
    return [int.from_bytes(b[i:i + 32], "little") for i in range(0, len(b), 32)]


def _put(w, pos, groups):
    """w[pos] = the groups' values one after the other, (value limbs, members) each."""
    k = 0
    for v, m in groups:
        w[pos[k:k + m]] = v
        k += m
    assert k <= len(pos)
    return w


def _minus(v):
    return O.int_to_limbs((O.R - O.limbs_to_int(v)) % O.R)


def _witness(kind, n, rng):
    w = O.random_fr(n, rng)
    w[0] = O.fr_mont(1)
    pos = rng.permutation(np.arange(1, n))
    v = O.random_fr(4400, rng)
    if kind == "many":      # more classes of the least size than one prove takes, smaller groups
        g = [(v[j], 4) for j in range(4200)] + [(v[j], 3) for j in range(4200, 4300)]
        # large classes (several fix-up levels), values beside their negations, zeros
        g += [(v[j], 500) for j in range(4300, 4310)]
        for j in range(4310, 4320):
            g += [(v[j], 8), (_minus(v[j]), 8)]
        return _put(w, pos, g + [(0 * v[0], 2000)])
    if kind == "few":       # most variables in two classes, one the negation of the other
        return _put(w, pos, [(v[0], n // 2), (_minus(v[0]), n // 3), (O.fr_mont(1), n // 8)])
    if kind == "equal":     # one class
        w[:] = O.fr_mont(O.R - 2)
        return w
    assert kind == "distinct"
    return w


KINDS = ("many", "few", "equal", "distinct")


@pytest.fixture(scope="module")
def keyed(ctx, orc):
    """A key of 2^17 variables, its discrete logs and one witness of each kind with the
    witness MSMs' points."""
    r1 = nk.generate("matmul", 40, 0, seed=31)
    assert r1.cols > 1 << 16
    tox = O.random_fr(5, np.random.default_rng(78))
    pk, _ = nk.setup(ctx, r1, tox)
    at, bt, lt, _, _ = orc.setup_scalars(r1, list(tox))
    logs = {"ar": (1, _ints(at)), "bs1": (1, _ints(bt)), "zk": (1, _ints(lt)), "bs2": (2, _ints(bt))}
    gens = {1: orc.g1_generator(), 2: orc.g2_generator()}
    rng = np.random.default_rng(79)
    cases = []
    for kind in KINDS:
        w = _witness(kind, r1.cols, rng)
        wi = _ints(w)
        want = {}
        for field, (group, k) in logs.items():
            total = sum(a * b for a, b in zip(wi, k)) * RINV % O.R  # Montgomery form
            want[field] = O.affine_to_jac(group, orc.mul_affine(group, gens[group], O.int_to_limbs(total)))[0]
        cases.append((w, want))
    be = nk.Backend(ctx)
    be.prepare(r1, pk)
    yield be, cases
    be.free()


def _check(raw, want, what):
    for field, point in want.items():
        assert np.array_equal(np.frombuffer(bytes(getattr(raw, field)), np.uint64), point), (field, what)


def test_single_proves(keyed):
    be, cases = keyed
    for i in (0, 1, 2, 3, 1, 0): # issued, captured, replayed
        _check(be.prove(cases[i][0]), cases[i][1], KINDS[i])


@pytest.mark.parametrize("lists", [False, True])
def test_batches_over_several_slots(keyed, lists):
    be, cases = keyed
    order = [0, 1, 2, 3, 3, 2, 0, 1, 0]
    for _ in range(2):
        raws = nk.prove_batch([be] * len(order), [cases[i][0] for i in order], lists=lists)
        for i, raw in zip(order, raws):
            _check(raw, cases[i][1], KINDS[i])
    assert len({bytes(raws[j].qz) for j, i in enumerate(order) if i == 0}) == 1


def test_server(ctx, keyed):
    be, cases = keyed
    sv = nk.Server(ctx, max_inflight=4, max_slots_per_key=3)
    kid = sv.add_key(be)
    order = [0, 1, 2, 3, 2, 1, 0, 3]
    rids = [(i, sv.submit(kid, cases[i][0])) for i in order]
    for i, rid in rids:
        _check(sv.wait(rid)[0], cases[i][1], KINDS[i])
    assert sv.slots(kid) > 1
    sv.close()
