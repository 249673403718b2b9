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


def test_threads_with_keys_of_their_own(ctx, orc):
    """Four threads prove and blind on a key each, from the first prove over the capture to
    replays, while this one allocates and runs MSMs and transforms on the same context."""
    import threading
    specs = [("poseidon", 2), ("poseidon", 20), ("matmul", 8), ("sql-aggregate", 8)]
    keys, want = [], []
    r, s = O.random_fr(2, np.random.default_rng(44))
    for kind, param in specs:
        r1, pk, be = _key(ctx, kind, param)
        one = nk.Backend(ctx)
        one.prepare(r1, pk)
        raw = one.prove(r1.witness)
        want.append((bytes(raw), bytes(one.blind(raw, r, s))))
        one.free()
        keys.append((be, r1.witness))
    bad = []

    def work(j):
        be, w = keys[j]
        try:
            for i in range(8):
                raw = be.prove(w)
                if (bytes(raw), bytes(be.blind(raw, r, s))) != want[j]:
                    bad.append((j, i))
        except Exception as e:
            bad.append((j, repr(e)))

    rng = np.random.default_rng(45)
    x, jac = O.random_fr(1 << 12, rng), np.tile(O.affine_to_jac(1, orc.g1_generator()[None]), (500, 1))
    sc = O.random_fr(500, rng)
    fft, msm = ctx.ntt(0, x), ctx.msm(1, jac, sc)
    threads = [threading.Thread(target=work, args=(j,)) for j in range(4)]
    for t in threads:
        t.start()
    while any(t.is_alive() for t in threads):
        assert np.array_equal(ctx.ntt(0, x), fft) and np.array_equal(ctx.msm(1, jac, sc), msm)
    for t in threads:
        t.join()
    assert not bad
    for be, _ in keys:
        be.free()
