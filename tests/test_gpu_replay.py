"""A key's first prove issues its launches, the second captures them into a graph and the
later ones replay it.  Whichever way a prove runs, and with batches on the same slot
between, the raw proofs, the blindings of present and earlier proofs and the stage times
are those of the issued prove."""
import numpy as np
import pytest

import nkr_b200 as nk
import oracle as O

pytestmark = pytest.mark.gpu


def _key(ctx, kind, param):
    r1 = nk.generate(kind, param, 1, seed=41)
    pk, _ = nk.setup(ctx, r1, O.random_fr(5, np.random.default_rng(42)))
    be = nk.Backend(ctx)
    be.prepare(r1, pk)
    return r1, pk, be


def _witnesses(kind, param, count):
    return [nk.generate(kind, param, 1, seed=50 + i).witness for i in range(count)]


def _affine(raw):
    g1, g2 = nk.raw_to_arrays(raw)
    return np.stack([x[:8] for x in g1]), g2[:16]


@pytest.mark.parametrize("kind,param", [("poseidon", 2), ("poseidon", 150)])
def test_replayed_proves_batches_and_blinding(ctx, orc, kind, param):
    """poseidon 2 has no class path, poseidon 150 (2^17 variables) has."""
    r1, pk, be = _key(ctx, kind, param)
    ws = _witnesses(kind, param, 4)
    want = []
    for w in ws: # a fresh key's first prove is issued
        one = nk.Backend(ctx)
        one.prepare(r1, pk)
        want.append(bytes(one.prove(w)))
        one.free()
    assert len(set(want)) == 4
    pka = O.pk_affine(pk, orc)
    r, s = O.random_fr(2, np.random.default_rng(43))

    def blind(raw):
        a, b, c = orc.blind(pka, *_affine(raw), r, s)
        got = be.blind(raw, r, s)
        for x, group, y in ((got.a, 1, a), (got.b, 2, b), (got.c, 1, c)):
            assert np.array_equal(np.frombuffer(bytes(x), np.uint64), O.affine_to_jac(group, y)[0])

    first = be.prove(ws[0])                        # issued
    assert bytes(first) == want[0]
    assert bytes(be.prove(ws[1])) == want[1]       # captured
    blind(first)                                   # not the proof whose tables the slot holds
    for lists in (False, True):
        out = nk.prove_batch([be] * 5, [ws[i] for i in (2, 3, 0, 1, 2)], lists=lists)
        assert [bytes(x) for x in out] == [want[i] for i in (2, 3, 0, 1, 2)]
        raw = be.prove(ws[3])                      # replayed after a batch on the same slot
        assert bytes(raw) == want[3]
        blind(raw)
        blind(first)
    assert [bytes(be.prove(w)) for w in ws] == want
    be.free()


@pytest.mark.parametrize("kind,param", [("poseidon", 2), ("poseidon", 150)])
def test_stage_times_of_issued_and_replayed_proves(ctx, kind, param):
    """Each MSM's phases in order and within the prove, also for replays, whose events are
    nodes of the graph, and after a batch, which records none."""
    r1, pk, be = _key(ctx, kind, param)
    w = _witnesses(kind, param, 1)[0]
    seen = []
    for i in range(6):
        be.prove(w)
        t = be.stage_times()
        seen.append(tuple(t.values()))
        slack = 1e-3 # the events' resolution
        for m in ("a", "b_g1", "b_g2", "l", "h"):
            order = [0.0] + [t[f"msm_{m}_{p}_ms"] for p in ("l1_start", "l1_end", "fixup_end", "reduce_first_end")]
            order += [t[f"msm_{m}_end_ms"], t["total_ms"]]
            assert all(x <= y + slack for x, y in zip(order, order[1:])), (i, m, order)
            assert order[2] > order[1]
        assert min(t["spmv_ms"], t["quotient_ms"], t["quotient_msm_ms"]) > 0
        assert t["spmv_ms"] + t["quotient_ms"] + t["quotient_msm_ms"] <= t["total_ms"] + 3 * slack
        assert abs(t["witness_msms_ms"] + t["spmv_ms"] - t["total_ms"]) < slack
        if i == 3:
            nk.prove_batch([be] * 2, [w] * 2)
            assert tuple(be.stage_times().values()) == seen[-1]
    assert len(set(seen)) == 6  # every prove's own
    be.free()
